// eq_tc.cu -- equalize + demodulate on the 5th-generation tensor cores.
//
// The mixed-precision replacement of the reference's SIMT equalizer
// (sgemv/equalize_kernel.cuh:27-481).  A CTA takes one subcarrier group g
// and up to 128 / sg of the launch's symbols, and computes the real-block
// GEMM
//     D (128 x N) = Y (128 x 2*Mp) * A_g^T (2*Mp x N),   N = 2K padded to 16,
// with BF16 operands and FP32 accumulation in tensor memory:
//   Y   = the planar BF16 FFT output y_lp[sym][plane][b][s], one row per
//         (symbol, subcarrier) column of the group, reduction index
//         kk = plane*Mp + b; MN-major in shared memory (each 8 x 16-byte
//         core matrix is 8 antennas x 8 consecutive subcarriers, one tensor
//         box of 8 subcarriers x 64 antennas per 1 KB);
//   A_g = R(W_g^T) with rows interleaved (2u: real part of user u, 2u+1:
//         imaginary part); the ZF kernel writes it into global memory already
//         in the shared-memory image of the K-major no-swizzle canonical
//         layout, one 64-wide k tile at a time, so one bulk copy per tile
//         stages it.
// D row i sits in TMEM lane i: every thread of the epilogue owns one
// (symbol, subcarrier) and reads the complex x of all K users from its own
// lane, demaps each (modulation/demodulation.h:30-67 in FP16), and stores the
// LLRs, so that consecutive lanes write consecutive stretches of each user's
// LLR row.  Hard bits of 8 neighbouring subcarriers are gathered with three
// shuffles into whole descrambled bytes.
//
// Pipeline: kStages shared-memory stages fed by one producer thread (bulk
// copy + tensor boxes); one thread issues the 4 MMAs per tile and commits
// them to the stage's mbarrier.  Every wait is bounded in time and reports a
// timeout through the device error word.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "eq_tc.cuh"
#include "eq_tc_epi.cuh"
#include "sgemv.cuh"
#include "tc.cuh"

namespace mb {

namespace {
constexpr int kStages = 3;  // at most; two k tiles (up to 64 antennas) take two stages
constexpr int kKT = 64;     // reduction elements per k tile (4 MMAs of K=16)
constexpr int kCols = 128;  // MMA M: (symbol, subcarrier) columns per CTA
constexpr int kEqThreads = 256;  // 8 warps: warps w and w + 4 read TMEM lane quadrant w
}  // namespace

template <int MM, int QM>
__global__ void __launch_bounds__(kEqThreads, 1)
    equalize_tc_kernel(const EqTcParams q, const __grid_constant__ CUtensorMap ymap) {
  extern __shared__ __align__(1024) uint8_t eq_smem[];
  pdl_wait();
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int timed_out;

  const EqParams &p = q.p;
  const uint32_t g = blockIdx.x;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  // this CTA's symbols: l_off .. l_off + nbc - 1 of the launch
  const uint32_t l_off = blockIdx.y * q.spc;
  const uint32_t nbc = min(q.spc, q.nb - l_off);
  const uint32_t ncols = nbc * p.sg;                 // valid columns, <= 128
  constexpr uint32_t y_tile = kCols * kKT * 2;       // 16 KB: 128 columns x 64 kk
  constexpr uint32_t a_tile = MM * kKT * 2;          // detector image k tile
  constexpr uint32_t stage_bytes = y_tile + a_tile;
  const uint32_t y_bytes = ncols * kKT * 2;          // bytes this CTA loads per tile
  const uint32_t s_base = g * p.sg;

  if (tid == 0) {
    for (int s = 0; s < kStages; s++) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
    tc::mbar_init(&done_bar, 1);
    tc::fence_mbar_init();
    timed_out = 0;
    tc::prefetch_tmap(&ymap);
  }
  if (warp == 0) tc::tmem_alloc(&tmem_base_slot, q.tmem_cols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base_slot;

  if (warp == 0 && lane == 0) {
    // ---- producer: y columns by tensor boxes, detector image by bulk copy
    const uint8_t *a_g = q.a_img + (uint64_t)g * q.nkt * a_tile;
    for (uint32_t kt = 0, s = 0, use = 0; kt < q.nkt; kt++) {
      if (use >= 1 && !tc::mbar_wait(&empty_bar[s], (use - 1) & 1)) {
        timed_out = 1;
        break;
      }
      uint8_t *sy = eq_smem + s * stage_bytes;
      uint8_t *sa = sy + y_tile;
      tc::mbar_arrive_expect_tx(&full_bar[s], y_bytes + a_tile);
      tc::bulk_g2s(sa, a_g + (uint64_t)kt * a_tile, a_tile, &full_bar[s]);
      const uint32_t kk0 = kt * kKT, plane = kk0 / q.Mp, b0 = kk0 % q.Mp;
      // boxes of 16 (swizzled, 2 KB) or 8 (1 KB) columns by the 64 k rows
      const uint32_t bw = q.y16 ? 16 : 8;
      for (uint32_t j = 0; j < ncols / bw; j++) {
        const uint32_t col0 = j * bw, l = col0 / p.sg, sl = col0 % p.sg;
        const int32_t row = (int32_t)(((l_off + l) * 2 + plane) * p.M + b0);
        tc::tma_load_2d(sy + j * bw * 128, &ymap, (int32_t)(s_base + sl), row, &full_bar[s]);
      }
      if (++s == q.stages) s = 0, use++;
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer.  Columns ncols..127 of the y stage are never loaded:
    // their D rows are garbage and no thread stores them.
    const uint32_t idesc = tc::idesc_bf16(kCols, q.N, true, false);
    bool ok = true;
    for (uint32_t kt = 0, s = 0, use = 0; kt < q.nkt; kt++) {
      if (!tc::mbar_wait(&full_bar[s], use & 1)) {
        ok = false;
        break;
      }
      tc::fence_after_sync();
      const uint32_t y0 = tc::smem_u32(eq_smem + s * stage_bytes), a0 = y0 + y_tile;
#pragma unroll
      for (int ks = 0; ks < kKT / 16; ks++) {
        // Y: MN-major.  8-column boxes: 8-antenna K groups 128 B apart,
        // 8-subcarrier MN chunks 1024 B apart (one box each); 16-column
        // swizzled boxes: 32-byte atoms of 16 columns 2048 B apart (one box
        // each), 8-antenna K groups 256 B apart
        const uint64_t yd = q.y16 ? tc::smem_desc_mn_sw32(y0 + ks * 512, 2048, 256)
                                  : tc::smem_desc(y0 + ks * 256, 128, 1024);
        // image: K-major, K core matrices 128 B apart, 8-row groups 1024 B apart
        const uint64_t ad = tc::smem_desc(a0 + ks * 256, 128, 1024);
        tc::mma_f16(tmem, yd, ad, idesc, (kt | ks) != 0);
      }
      tc::mma_commit(&empty_bar[s]);
      if (++s == q.stages) s = 0, use++;
    }
    if (ok) tc::mma_commit(&done_bar);
    else timed_out = 1;
  }
  __syncwarp();
  // the epilogue's per-thread setup overlaps the load/MMA phase
  EqTcEpilogue<MM, QM> epi;
  epi.prepare(p, s_base, l_off, ncols, q.l0, q.N, warp, lane);
  // everyone: wait for the accumulator (bounded)
  bool ok = tc::mbar_wait(&done_bar, 0);
  if (__syncthreads_or(!ok || timed_out)) {
    if (tid == 0 && q.err) atomicOr(q.err, tc::kErrTimeout);
  } else {
    tc::fence_after_sync();
    epi.run(p, tmem, warp, lane);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, q.tmem_cols);
}

TcShape tc_shape(uint32_t M, uint32_t K) {
  TcShape s;
  s.MM = 2 * K <= 64 ? 64 : 128;
  s.Mp = (M + kKT - 1) / kKT * kKT;
  s.nkt = 2 * s.Mp / kKT;
  s.img_group_bytes = (uint64_t)s.nkt * s.MM * kKT * 2;
  return s;
}

using EqTcKernel = void (*)(const EqTcParams, const CUtensorMap);

template <int MM>
static EqTcKernel eq_tc_kernel_of(uint32_t Qm) {
  switch (Qm) {
    case 2: return equalize_tc_kernel<MM, 2>;
    case 4: return equalize_tc_kernel<MM, 4>;
    case 6: return equalize_tc_kernel<MM, 6>;
    default: return equalize_tc_kernel<MM, 8>;
  }
}

// raises the dynamic shared memory limit of the (MM, Qm) kernel once per device
static mb_status equalize_tc_configure(uint32_t MM, uint32_t Qm, int dev) {
  static std::atomic<uint64_t> configured[8] = {};
  const int which = (MM == 64 ? 0 : 4) + (Qm == 2 ? 0 : Qm == 4 ? 1 : Qm == 6 ? 2 : 3);
  const uint64_t bit = 1ull << (dev & 63);
  if (configured[which].load() & bit) return MB_OK;
  int maxs = 0;
  MB_CUDA_TRY(cudaDeviceGetAttribute(&maxs, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const EqTcKernel k = MM == 64 ? eq_tc_kernel_of<64>(Qm) : eq_tc_kernel_of<128>(Qm);
  cudaFuncAttributes fa;
  MB_CUDA_TRY(cudaFuncGetAttributes(&fa, k));
  MB_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   maxs - (int)fa.sharedSizeBytes));
  configured[which].fetch_or(bit);
  return MB_OK;
}

bool equalize_tc_supported(uint32_t K, uint32_t sg, uint32_t nb) {
  // a CTA holds whole symbols of one group in its 128 columns; the MMA's N
  // is 2K rounded up to 16 (at most the image's MM rows)
  if (K == 0 || K > 64 || sg == 0 || sg % 8 != 0 || sg > (uint32_t)kCols) return false;
  return nb >= 1;
}

mb_status equalize_tc(const EqParams &p, const void *a_img, const void *y_lp, uint32_t S_pad,
                      uint32_t l0, uint32_t nb, int *err, cudaStream_t st, uint32_t max_cols) {
  if (!equalize_tc_supported(p.K, p.sg, nb)) return MB_UNSUPPORTED;
  if (S_pad % 8 || S_pad < p.S) return MB_BAD_SHAPE;
  TcShape s = tc_shape(p.M, p.K);
  EqTcParams q;
  q.p = p;
  q.a_img = reinterpret_cast<const uint8_t *>(a_img);
  q.y_lp = reinterpret_cast<const __nv_bfloat16 *>(y_lp);
  q.S_pad = S_pad;
  q.Mp = s.Mp;
  q.nkt = s.nkt;
  // symbols per CTA: as many as fill max_cols (<= 128) columns, spread
  // evenly over the CTAs a group needs
  const uint32_t cols = max_cols ? std::min<uint32_t>(max_cols, kCols) : kCols;
  const uint32_t spc_max = std::max<uint32_t>(1, cols / p.sg);
  const uint32_t ny = (nb + spc_max - 1) / spc_max;
  q.spc = (nb + ny - 1) / ny;
  q.nb = nb;
  q.N = (2 * p.K + 15) / 16 * 16;
  q.l0 = l0;
  q.err = err;
  q.tmem_cols = 32;
  while (q.tmem_cols < q.N) q.tmem_cols *= 2;
  // two k tiles need no third stage: 48 instead of 72 KB (MM = 64), four
  // CTAs per SM instead of three (32 uneven cells, most of up to 64 antennas:
  // 547 -> 533 us a slot of each)
  q.stages = std::min<uint32_t>(kStages, s.nkt);
  const size_t smem = (size_t)q.stages * ((size_t)kCols * kKT * 2 + (size_t)s.MM * kKT * 2);
  const uint32_t G = (p.S + p.sg - 1) / p.sg;
  int dev = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  mb_status cs = equalize_tc_configure(s.MM, p.Qm, dev);
  if (cs != MB_OK) return cs;
  // tensor map over y_lp rows [nb * 2 * M][S_pad], box 16 subcarriers x 64
  // antennas with the 32-byte swizzle (one 2 KB MN-major SW32 atom column:
  // whole 32-byte sectors per antenna row) when groups are whole boxes, else
  // 8 subcarriers x 64 antennas (one 1 KB group of MN-major core matrices)
  q.y16 = p.sg % 16 == 0 ? 1 : 0;
  CUtensorMap ymap;
  mb_status tr = make_tmap_2d_bf16(&ymap, y_lp, S_pad, (uint64_t)nb * 2 * p.M, S_pad, q.y16 ? 16 : 8, kKT,
                                   q.y16 != 0);
  if (tr != MB_OK) return tr;
  const dim3 grid(G, ny);
  MB_CUDA_TRY(pdl_launch(s.MM == 64 ? eq_tc_kernel_of<64>(p.Qm) : eq_tc_kernel_of<128>(p.Qm), grid, kEqThreads, smem,
                         st, q, ymap));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

}  // namespace mb

namespace mb {

// ---- the same GEMM from FP32 operands (mb_equalize_tc) -------------------
// W [G][M][K] and y [sym][M][S] are read once, as they are, and rounded to
// BF16 on their way into shared memory: the images and planar rows that the
// slot's FFT and ZF kernels prepare do not exist here, and writing them first
// moved 107 MB more at the 256 x 32 cell (12 symbols, 3276 subcarriers) in two
// more launches.  DRAM bound: 94 MB of operands and 16 MB of results there.
// The 256 threads hold the next 32 antennas of both operands in registers
// (about 32 KB of loads in flight per CTA, three CTAs per SM) while the tensor
// core multiplies the previous two tiles.  One call there: 130 us with
// the three launches, 29 us with this one (kernel 26 us, 4.2 TB/s).
// Layouts per tile (32 antennas, planes re and im one after the other):
//   Y: MN-major, core matrices of 8 antennas x 8 columns, antenna groups 128 B
//      apart, column chunks kTSbo apart;
//   A: K-major, rows 2u / 2u + 1 the real and imaginary part of user u, k
//      core matrices 128 B apart, 8-row groups kTSbo apart.
// kTSbo is 512 + 16 bytes so that lanes that store neighbouring chunks or row
// groups meet different banks.  Rows past 2K of A and columns past ncols of Y
// hold leftovers: they only reach accumulators that nothing reads.
constexpr int kTA = 32;           // antennas per tile
constexpr uint32_t kTSbo = 528;
constexpr int kYUnits = 8;        // column pairs per thread and tile, at most
constexpr uint32_t kTY = 16 * kTSbo;  // one plane of Y

template <int MM, int QM>
__global__ void __launch_bounds__(kEqThreads, MM == 64 ? 3 : 2)
    equalize_tc_c32_kernel(const EqParams p, uint32_t l0, uint32_t nb, uint32_t spc, uint32_t N,
                           uint32_t tmem_cols, uint32_t vw_log2, uint32_t vec, int *err) {
  extern __shared__ __align__(128) uint8_t ec_smem[];
  pdl_wait();
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tmem_base_slot;
  constexpr uint32_t a_plane = MM / 8 * kTSbo, stage_bytes = 2 * kTY + 2 * a_plane;
  constexpr uint32_t KP = MM / 2;  // users a tile has room for
  const uint32_t g = blockIdx.x, tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const uint32_t l_off = blockIdx.y * spc, nbc = min(spc, nb - l_off), ncols = nbc * p.sg;
  const uint32_t s_base = g * p.sg;
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(&tmem_base_slot, tmem_cols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base_slot;

  // y: this thread's column pair v of the tile's antennas yb, yb + ystep, ...
  const uint32_t v = tid & ((1u << vw_log2) - 1), yb = tid >> vw_log2, ystep = kEqThreads >> vw_log2;
  const uint32_t c = 2 * v, l = c / p.sg, s = s_base + c - l * p.sg;
  const bool y0_on = c < ncols && s < p.S, y1_on = c < ncols && s + 1 < p.S;
  const float2 *yp = p.y + ((uint64_t)(l0 + l_off + l) * p.M + yb) * p.S + s;
  const uint32_t y_dst = (v / 4) * kTSbo + (v % 4) * 4 + yb * 16;  // antenna b of a chunk: 16 b bytes on
  // W: user u, the tile's antennas 8 kc .. 8 kc + 7
  const uint32_t u = tid % KP, kc = tid / KP;
  const bool w_on = kc < kTA / 8 && u < p.K;
  const float2 *wp = p.W + ((uint64_t)g * p.M + 8 * kc) * p.K + u;
  const uint32_t a_dst = 2 * kTY + (u / 4) * kTSbo + (2 * u % 8) * 16 + kc * 128;

  float4 yr[kYUnits];
  float2 wr[8];
  // the next tile's operands (yp and wp move on with it): antennas left of M
  // rows remain; a whole tile needs no look at the single rows
  const uint64_t ys = (uint64_t)ystep * p.S;
  const uint32_t nyu = kTA / ystep;  // column pairs per thread (uniform)
  auto load_rows = [&](uint32_t left, auto whole) {
    constexpr bool kWhole = decltype(whole)::value;
    const float2 *q = yp;
#pragma unroll
    for (int j = 0; j < kYUnits; j++) {
      yr[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j < (int)nyu && (kWhole || yb + j * ystep < left)) {
        if (vec && y1_on) {
          yr[j] = *reinterpret_cast<const float4 *>(q);
        } else {
          if (y0_on) *reinterpret_cast<float2 *>(&yr[j].x) = *q;
          if (y1_on) *reinterpret_cast<float2 *>(&yr[j].z) = q[1];
        }
      }
      q += ys;
    }
    const float2 *w = wp;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      wr[j] = make_float2(0.f, 0.f);
      if (w_on && (kWhole || 8 * kc + j < left)) wr[j] = *w;
      w += p.K;
    }
    yp += (uint64_t)kTA * p.S;
    wp += (uint64_t)kTA * p.K;
  };
  auto load = [&](uint32_t b0) {
    if (b0 + kTA <= p.M) load_rows(kTA, std::true_type{});
    else load_rows(p.M - b0, std::false_type{});
  };
  auto pack = [](float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
  };
  auto store = [&](uint8_t *st) {
    if (c < ncols) {
#pragma unroll
      for (int j = 0; j < kYUnits; j++) {
        if (j >= (int)nyu) break;
        uint8_t *d = st + y_dst + j * ystep * 16;
        *reinterpret_cast<uint32_t *>(d) = pack(yr[j].x, yr[j].z);
        *reinterpret_cast<uint32_t *>(d + kTY) = pack(yr[j].y, yr[j].w);
      }
    }
    if (w_on) {
      uint4 re, im, ng;
      re = make_uint4(pack(wr[0].x, wr[1].x), pack(wr[2].x, wr[3].x), pack(wr[4].x, wr[5].x), pack(wr[6].x, wr[7].x));
      im = make_uint4(pack(wr[0].y, wr[1].y), pack(wr[2].y, wr[3].y), pack(wr[4].y, wr[5].y), pack(wr[6].y, wr[7].y));
      ng = make_uint4(im.x ^ 0x80008000u, im.y ^ 0x80008000u, im.z ^ 0x80008000u, im.w ^ 0x80008000u);
      uint8_t *d = st + a_dst;
      *reinterpret_cast<uint4 *>(d) = re;                  // x.re = W.re y.re - W.im y.im
      *reinterpret_cast<uint4 *>(d + 16) = im;             // x.im = W.im y.re + W.re y.im
      *reinterpret_cast<uint4 *>(d + a_plane) = ng;
      *reinterpret_cast<uint4 *>(d + a_plane + 16) = re;
    }
  };

  const uint32_t idesc = tc::idesc_bf16(kCols, N, true, false);
  const uint32_t nt = (p.M + kTA - 1) / kTA;
  bool ok = true;
  load(0);
  for (uint32_t t = 0; t < nt; t++) {
    const uint32_t sidx = t & 1;
    // the stage's previous tile (t - 2) must have been multiplied
    if (t >= 2 && !tc::mbar_wait(&bar[sidx], ((t - 2) >> 1) & 1)) ok = false;
    uint8_t *st = ec_smem + sidx * stage_bytes;
    store(st);
    if (t + 1 < nt) load((t + 1) * kTA);
    tc::fence_proxy_async_smem();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    if (tid == 0) {
      tc::fence_after_sync();
      const uint32_t y0 = tc::smem_u32(st), a0 = y0 + 2 * kTY;
#pragma unroll
      for (int k = 0; k < 2 * (kTA / 16); k++) {
        const uint32_t pl = k / (kTA / 16), ks = k % (kTA / 16);
        tc::mma_f16(tmem, tc::smem_desc(y0 + pl * kTY + ks * 256, 128, kTSbo),
                    tc::smem_desc(a0 + pl * a_plane + ks * 256, 128, kTSbo), idesc, (t | k) != 0);
      }
      tc::mma_commit(&bar[sidx]);
    }
  }
  // the epilogue's per-thread setup overlaps the last MMAs
  EqTcEpilogue<MM, QM> epi;
  epi.prepare(p, s_base, l_off, ncols, l0, N, warp, lane);
  // the last tile's commit covers every MMA issued before it
  if (ok && !tc::mbar_wait(&bar[(nt - 1) & 1], ((nt - 1) >> 1) & 1)) ok = false;
  if (__syncthreads_or(!ok)) {
    if (tid == 0 && err) atomicOr(err, tc::kErrTimeout);
  } else {
    tc::fence_after_sync();
    epi.run(p, tmem, warp, lane);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, tmem_cols);
}

template <int MM>
static void eq_tc_c32_launch(const EqParams &p, uint32_t l0, uint32_t nb, int *err, cudaStream_t st, bool configure,
                             cudaError_t *e) {
  constexpr size_t smem = 2 * (2 * (size_t)kTY + 2 * MM / 8 * (size_t)kTSbo);
  auto k = p.Qm == 2   ? equalize_tc_c32_kernel<MM, 2>
           : p.Qm == 4 ? equalize_tc_c32_kernel<MM, 4>
           : p.Qm == 6 ? equalize_tc_c32_kernel<MM, 6>
                       : equalize_tc_c32_kernel<MM, 8>;
  if (configure) {
    *e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return;
  }
  const uint32_t N = (2 * p.K + 15) / 16 * 16;
  uint32_t tmem_cols = 32;
  while (tmem_cols < N) tmem_cols *= 2;
  // symbols per CTA: as many as fill the 128 columns, spread evenly over the
  // CTAs a group needs
  const uint32_t spc_max = std::max<uint32_t>(1, kCols / p.sg), ny = (nb + spc_max - 1) / spc_max;
  const uint32_t spc = (nb + ny - 1) / ny;
  // column pairs side by side in the 256 threads: a power of two, at least
  // the 8 with which the threads cover a tile's 32 antennas in one pass
  uint32_t vw = 3;
  while ((2u << vw) < spc * p.sg) vw++;
  const uint32_t vec = p.S % 2 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
  const dim3 grid((p.S + p.sg - 1) / p.sg, ny);
  *e = pdl_launch(k, grid, kEqThreads, smem, st, p, l0, nb, spc, N, tmem_cols, vw, vec, err);
}

mb_status equalize_tc_c32(const EqParams &p, int *err, cudaStream_t st) {
  if (!equalize_tc_supported(p.K, p.sg, 1)) return MB_UNSUPPORTED;
  auto launch = p.K <= 32 ? eq_tc_c32_launch<64> : eq_tc_c32_launch<128>;
  static std::atomic<uint64_t> configured[8] = {};
  const int which = (p.K <= 32 ? 0 : 4) + (int)p.Qm / 2 - 1;
  int dev = 0;
  cudaError_t e = cudaSuccess;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured[which].load() & bit)) {
    launch(p, 0, 0, err, st, true, &e);
    MB_CUDA_TRY(e);
    configured[which].fetch_or(bit);
  }
  constexpr uint32_t kMaxSyms = 32768;  // grid.y's range
  for (uint32_t l0 = 0; l0 < p.n_sym; l0 += kMaxSyms) {
    launch(p, l0, std::min(kMaxSyms, p.n_sym - l0), err, st, false, &e);
    MB_CUDA_TRY(e);
  }
  return MB_OK;
}

}  // namespace mb

using namespace mb;

extern "C" mb_status mb_equalize_tc_scratch(uint32_t K, uint32_t M, uint32_t S, uint32_t sg,
                                            uint32_t n_sym, uint64_t *img_bytes,
                                            uint64_t *ylp_bytes) {
  if (!img_bytes || !ylp_bytes) return MB_BAD_ARG;
  if (K == 0 || K > 64 || M == 0 || S == 0 || sg == 0) return MB_BAD_SHAPE;
  // W and y are rounded on their way into shared memory: what is left of the
  // images and planar rows that stood here is that the pointers are not NULL
  *img_bytes = 16;
  *ylp_bytes = n_sym ? 16 : 0;
  return MB_OK;
}

extern "C" mb_status mb_equalize_tc(const mb_c32 *W, const mb_c32 *y, uint32_t K, uint32_t M,
                                    uint32_t S, uint32_t sg, uint32_t n_sym, uint32_t Qm,
                                    uint64_t cb_size, uint64_t cb_stride, uint64_t zeros,
                                    uint32_t cb_blocks, uint16_t *llr, uint8_t *hard,
                                    const mb_scrambler *scr, mb_c32 *x, void *scratch_img,
                                    void *scratch_ylp, void *stream) {
  EqParams p;
  mb_status s = equalize_prepare(p, W, y, K, M, S, sg, n_sym, Qm, cb_size, cb_stride, zeros,
                                 cb_blocks, llr, hard, scr);
  if (s != MB_OK) return s;
  if (!scratch_img || !scratch_ylp) return MB_BAD_ARG;
  p.x = reinterpret_cast<float2 *>(x);
  if (n_sym == 0) return MB_OK;
  if (!equalize_tc_supported(K, sg, 1)) return MB_UNSUPPORTED;
  const DeviceTables *tab = device_tables();
  if (!tab) return MB_CUDA_ERROR;
  return equalize_tc_c32(p, tab->err, as_stream(stream));
}
