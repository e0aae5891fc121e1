// mlp_step.cu -- forward, loss and backward pass of the 3-layer MLP in one
// kernel (see mlp.cu for the network, its loss and its rounding points).
//
// A product per launch leaves a training step latency bound: 17 launches of a
// few microseconds of arithmetic each.  Here a CTA takes 64 samples through
// all eight products of the step; activations and upstream gradients stay in
// shared memory as the BF16 operands the products take anyway, accumulators
// in tensor memory (FP32), and only the parameter gradients leave the CTA, as
// one slot of partial sums that a second kernel adds in slot order
// (deterministic).  Every product is laid out with neurons in the MMA's 128
// rows (a TMEM lane, i.e. a thread, owns neuron tid):
//   z1^T = W1^T x^T, z2^T = W2^T h1^T, dz2^T = W3 dy^T, dz1^T = W2 dz2^T
// (64 sample columns each), so biases, ReLU masks (64 bits a thread and
// layer) and the bias gradients (sums over a thread's own columns, FP32,
// before the rounding) need no exchange between threads.  All matrices sit in
// shared memory as 8 x 8 blocks of 128 bytes; such a block is a core matrix
// both of a K-major operand (k along its rows' 16 bytes) and of an MN-major
// one (k across its rows), so each serves every product it enters without a
// transposition.
// Eight steps of 22 -> 256 -> 256 -> 4 on batches of 4096 (with the host copies
// of gradients and weights at the end): 6,930 us with a product per launch, 400
// us here (25 us this kernel, 4.2 us the reduction, 2.8 us Adam per step, the
// rest the host's copies and launches).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "mlp_step.cuh"
#include "tc.cuh"

namespace mb {
namespace {

constexpr uint32_t kT = kStepTile;
constexpr uint32_t kH = kT / 8 * 128;  // bytes between the block rows of a [.][64] activation matrix

struct StepParams {
  MlpStepShape s;
  const __nv_bfloat16 *img;
  const float *params, *x, *A, *b, *c;
  float *part;
  int *err;
  uint32_t B, tiles;
  BlendFeatures f;  // inference without x
  float *y;         // inference: the outputs
};

// one operand: shared-memory address, leading and stride byte offsets, bytes
// from one K = 16 step to the next
struct Opnd {
  uint32_t a, lbo, sbo, step;
};
__device__ __forceinline__ void mma_steps(uint32_t d, const Opnd &A, const Opnd &B, uint32_t idesc, uint32_t ksteps) {
  for (uint32_t k = 0; k < ksteps; k++)
    tc::mma_f16(d, tc::smem_desc(A.a + k * A.step, A.lbo, A.sbo), tc::smem_desc(B.a + k * B.step, B.lbo, B.sbo),
                idesc, k != 0);
}
// k along the blocks' rows' 16 bytes / across their rows; rs: bytes between block rows
__device__ __forceinline__ Opnd kmajor(uint32_t a, uint32_t rs) { return {a, 128, rs, 256}; }
__device__ __forceinline__ Opnd mnmajor(uint32_t a, uint32_t rs) { return {a, rs, 128, 2 * rs}; }

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}
// 16 values of matrix row n, columns 16 c .. 16 c + 15, rounded to BF16
__device__ __forceinline__ void put16(uint8_t *m, uint32_t n, uint32_t c, const float *v) {
  uint8_t *d = m + n / 8 * kH + c * 256 + n % 8 * 16;
  *reinterpret_cast<uint4 *>(d) = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
  *reinterpret_cast<uint4 *>(d + 128) =
      make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]), pack2(v[14], v[15]));
}

// MT: 128-neuron tiles (width up to 128 MT), 128 MT threads.  FWD: inference,
// which ends with y (1200 samples of 22 -> 256 -> 256 -> 4: 32 us on the CUDA
// cores, 8.7 us here).
template <int MT, bool FWD>
__global__ void __launch_bounds__(128 * MT, 1) mlp_step_kernel(const StepParams q) {
  extern __shared__ __align__(1024) uint8_t st_smem[];
  pdl_wait();
  __shared__ __align__(8) uint64_t bar, bar_g, wbar1, wbar2;
  __shared__ uint32_t tmem_slot;
  __shared__ float red[2][kStepMaxOut + 1];
  constexpr uint32_t Wp = 128 * MT, nthr = 128 * MT;
  constexpr uint32_t rs2 = Wp / 8 * 128, rs3 = 256, rsd = 256;  // block rows of W1 / W2, W3, dy
  constexpr uint32_t w2_bytes = Wp * Wp * 2, h_bytes = Wp / 8 * kH;
  const MlpStepShape &s = q.s;
  const uint32_t I = s.I, W = s.W, O = s.O, Ip = s.Ip, rsx = Ip / 8 * 128;
  // W2 (dz1 once the products with W2 are done), h1, h2 (W1 before it, dz2
  // after it), x, W3, dy, then A, b and c of the tile for O <= 4
  uint8_t *w2 = st_smem, *h1 = w2 + w2_bytes, *h2 = h1 + h_bytes, *xs = h2 + h_bytes, *w3 = xs + kT * Ip * 2,
          *dy = w3 + Wp * 16 * 2;
  float *abc = reinterpret_cast<float *>(dy + kT * 16 * 2);
  const uint32_t a_w2 = tc::smem_u32(w2), a_h1 = tc::smem_u32(h1), a_h2 = tc::smem_u32(h2), a_x = tc::smem_u32(xs),
                 a_w3 = tc::smem_u32(w3), a_dy = tc::smem_u32(dy);
  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32, n = tid;
  const bool stage_abc = O <= 4;
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    tc::mbar_init(&bar_g, 1);
    tc::mbar_init(&wbar1, 1);
    tc::mbar_init(&wbar2, 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot, quad = (warp % 4) << 21, my = tmem + quad;
  // accumulators: z1 then dz2, z2 then dz1, y and dW3 (then dW2), dW1
  const uint32_t c_a = 0, c_b = 64 * MT, c_y = 256, c_w3 = 272, c_w2 = 256, c_w1 = 0;
  const uint32_t tl = warp / 4;  // this warp's 128-neuron tile
  constexpr uint32_t kB = 1;     // idesc flags: B MN-major
  const uint32_t id_z1 = tc::idesc_bf16(128, kT, true, false), id_z2 = tc::idesc_bf16(128, kT, true, kB),
                 id_y = tc::idesc_bf16(128, 16, true, kB), id_d2 = tc::idesc_bf16(128, kT, false, false),
                 id_w3 = tc::idesc_bf16(128, 16, false, kB), id_d1 = tc::idesc_bf16(128, kT, false, kB),
                 id_w2 = tc::idesc_bf16(128, Wp, false, false), id_w1 = tc::idesc_bf16(128, Ip, false, kB);
  const float bias1 = n < W ? q.params[s.off[1] + n] : 0.f, bias2 = n < W ? q.params[s.off[3] + n] : 0.f;
  float *slot = q.part + (uint64_t)blockIdx.x * s.slot;
  uint32_t ph = 0, ph_g = 0, pass = 0;
  bool ok = true;
  // every thread past the barrier's next phase (false: some wait gave up)
  auto arrived = [&](uint64_t *b, uint32_t &p) {
    const bool w = tc::mbar_wait(b, p & 1);
    p++;
    const bool all = !__syncthreads_or(!w);
    tc::fence_after_sync();
    return all;
  };
  // this thread's shared-memory writes and TMEM reads before the next MMAs
  auto publish = [&]() {
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  };
  // gradient element e of this CTA's slot: written by the first tile, added to by the others
  auto acc1 = [&](uint64_t e, float v) { slot[e] = pass ? slot[e] + v : v; };
  // ReLU layer: z columns at col + bias -> BF16 activations, sign mask.  The
  // loops over 16-column chunks stay loops: the kernel runs its code once, and
  // fetching it costs as much as running it
  auto hidden = [&](uint32_t col, float bias, uint8_t *h, uint32_t nv, uint64_t &mask) {
    mask = 0;
#pragma unroll 1
    for (uint32_t c = 0; c < 4; c++) {
      float v[16];
      tc::tmem_ld16(my + col + tl * kT + c * 16, v);
      uint32_t bits = 0;
#pragma unroll
      for (uint32_t j = 0; j < 16; j++) {
        const float z = v[j] + bias;
        if (z > 0.f) bits |= 1u << j;
        v[j] = 16 * c + j < nv ? fmaxf(z, 0.f) : 0.f;
      }
      mask |= (uint64_t)bits << (16 * c);
      put16(h, n, c, v);
    }
  };
  // upstream gradient: columns at col where the mask is set -> BF16, and their FP32 sum
  auto upstream = [&](uint32_t col, uint8_t *d, uint64_t mask) {
    float sum = 0.f;
#pragma unroll 1
    for (uint32_t c = 0; c < 4; c++) {
      float v[16];
      tc::tmem_ld16(my + col + tl * kT + c * 16, v);
      const uint32_t bits = (uint32_t)(mask >> (16 * c));
#pragma unroll
      for (uint32_t j = 0; j < 16; j++) {
        if (!(bits >> j & 1u)) v[j] = 0.f;
        sum += v[j];
      }
      put16(d, n, c, v);
    }
    return sum;
  };
  // dW2 columns 128 t .. 128 t + 127 (dW2^T = dz2^T h1: a thread holds 128
  // rows of one column) into the slot: a warp's lanes store neighbouring
  // columns of one row
  auto drain_w2 = [&](uint32_t t) {
    const uint32_t n2 = t * 128 + warp % 4 * 32 + lane, r0 = warp / 4 * 128;
#pragma unroll 1
    for (uint32_t r = r0; r < r0 + 128; r += 16) {
      float v[16];
      tc::tmem_ld16(my + c_w2 + r, v);
      if (n2 < W)
#pragma unroll
        for (uint32_t j = 0; j < 16; j++)
          if (r + j < W) acc1(s.off[2] + (uint64_t)(r + j) * W + n2, v[j]);
    }
  };

  for (uint32_t tile = blockIdx.x; tile < q.tiles; tile += gridDim.x, pass++) {
    const uint32_t row0 = tile * kT, nv = min(kT, q.B - row0);
    if (pass) publish();  // the previous tile's shared memory is about to be overwritten
    if (tid == 0) {
      tc::mbar_arrive_expect_tx(&wbar1, (Ip * Wp + Wp * 16) * 2);
      tc::bulk_g2s(h2, q.img, Ip * Wp * 2, &wbar1);  // W1
      tc::bulk_g2s(w3, q.img + s.img3(), Wp * 16 * 2, &wbar1);
      tc::mbar_arrive_expect_tx(&wbar2, w2_bytes);
      tc::bulk_g2s(w2, q.img + s.img2(), w2_bytes, &wbar2);
    }
    // inference on features: the six statistics of the tile's groups, a warp a
    // group, in the (unused) dy region
    float *fs = reinterpret_cast<float *>(dy);
    const uint32_t fg0 = FWD && !q.x ? row0 / q.f.sg : 0;
    if (FWD && !q.x) {
      const uint32_t KK = q.f.K * q.f.K;
      for (uint32_t g = fg0 + warp; g <= (row0 + nv - 1) / q.f.sg; g += nthr / 32) {
        const float2 *c0 = q.f.gc + (uint64_t)g * KK;
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // ||C_g||^2, trace, then distances and traces of j = -1, 1, 2
        for (uint32_t e = lane; e < KK; e += 32) {
          const float2 a = c0[e];
          const bool diag = e % (q.f.K + 1) == 0;
          v[0] += a.x * a.x + a.y * a.y;
          if (diag) v[1] += a.x;
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const int gj = (int)g + (k == 0 ? -1 : k);
            if (gj < 0 || gj >= (int)q.f.G) continue;
            const float2 b = q.f.gc[(uint64_t)gj * KK + e];
            v[2 + k] += (b.x - a.x) * (b.x - a.x) + (b.y - a.y) * (b.y - a.y);
            if (diag) v[5 + k] += b.x;
          }
        }
#pragma unroll
        for (int i = 0; i < 8; i++)
          for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if (lane < 3) {
          const int gj = (int)g + (lane == 0 ? -1 : (int)lane);
          const bool in = gj >= 0 && gj < (int)q.f.G;
          const float n0 = sqrtf(v[0]), d = lane == 0 ? v[2] : lane == 1 ? v[3] : v[4],
                      t = lane == 0 ? v[5] : lane == 1 ? v[6] : v[7];
          fs[(g - fg0) * 6 + lane] = in && n0 > 0.f ? sqrtf(d) / n0 : 0.f;
          fs[(g - fg0) * 6 + 3 + lane] = in && v[1] > 0.f ? t / v[1] - 1.f : 0.f;
        }
      }
      __syncthreads();
    }
    for (uint32_t e = tid; e < kT * (Ip / 8); e += nthr) {
      const uint32_t r = e / (Ip / 8), ch = e % (Ip / 8);
      float v[8];
#pragma unroll
      for (uint32_t j = 0; j < 8; j++) {
        const uint32_t f = ch * 8 + j, row = row0 + r;
        v[j] = 0.f;
        if (r < nv && f < I) {
          if (!FWD || q.x) v[j] = q.x[(uint64_t)row * I + f];
          else v[j] = f < q.f.sg ? (f == row % q.f.sg ? 1.f : 0.f) : fs[(row / q.f.sg - fg0) * 6 + f - q.f.sg];
        }
      }
      *reinterpret_cast<uint4 *>(xs + r / 8 * rsx + ch * 128 + r % 8 * 16) =
          make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
    }
    if (!FWD && stage_abc) {
      for (uint32_t e = tid; e < nv * O * O; e += nthr) abc[e] = q.A[(uint64_t)row0 * O * O + e];
      for (uint32_t e = tid; e < nv * O; e += nthr) abc[kT * 16 + e] = q.b[(uint64_t)row0 * O + e];
      for (uint32_t e = tid; e < nv; e += nthr) abc[kT * 20 + e] = q.c ? q.c[row0 + e] : 0.f;
    }
    if (!tc::mbar_wait(&wbar1, pass & 1)) ok = false;
    publish();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    uint64_t m1, m2;
    if (tid == 0) {
      for (uint32_t t = 0; t < MT; t++)
        mma_steps(tmem + c_a + t * kT, mnmajor(a_h2 + t * 2048, rs2), kmajor(a_x, rsx), id_z1, Ip / 16);
      tc::mma_commit(&bar);
    }
    if (!(ok = arrived(&bar, ph))) break;
    hidden(c_a, bias1, h1, nv, m1);
    if (!tc::mbar_wait(&wbar2, pass & 1)) ok = false;  // W2 has had the first layer to land
    publish();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    if (tid == 0) {
      for (uint32_t t = 0; t < MT; t++)
        mma_steps(tmem + c_b + t * kT, mnmajor(a_w2 + t * 2048, rs2), mnmajor(a_h1, kH), id_z2, Wp / 16);
      tc::mma_commit(&bar);
    }
    if (!(ok = arrived(&bar, ph))) break;
    hidden(c_b, bias2, h2, nv, m2);
    publish();
    if (tid == 0) {
      // rows 64..127 of the M = 128 operand are whatever follows: lanes never read
      mma_steps(tmem + c_y, mnmajor(a_h2, kH), mnmajor(a_w3, rs3), id_y, Wp / 16);
      tc::mma_commit(&bar);
    }
    if (!(ok = arrived(&bar, ph))) break;
    if (FWD) {
      if (warp < 2) {
        float y[16];
        tc::tmem_ld16(my + c_y, y);
        float *d = q.y + (uint64_t)(row0 + tid) * O;
        const float *b3 = q.params + s.off[5];
        if (tid < nv) {
#pragma unroll
          for (uint32_t r = 0; r < 16; r++)
            if (r < O) d[r] = y[r] + b3[r];
        }
      }
      continue;
    }
    if (warp < 2) {
      // sample tid: y, the loss and dy = 2 (A y - b) / B
      float y[16], g[16];
      tc::tmem_ld16(my + c_y, y);
      const bool in = tid < nv;
      const float *Ai = stage_abc ? abc + tid * O * O : q.A + (uint64_t)(row0 + (in ? tid : 0)) * O * O;
      const float *bi = stage_abc ? abc + kT * 16 + tid * O : q.b + (uint64_t)(row0 + (in ? tid : 0)) * O;
#pragma unroll
      for (uint32_t r = 0; r < 16; r++) {
        y[r] = r < O ? y[r] + q.params[s.off[5] + r] : 0.f;
        g[r] = 0.f;
      }
      float quad_y = 0.f, lin = 0.f;
      auto outputs = [&](auto om) {  // rows and columns up to om (>= O)
        constexpr uint32_t OM = decltype(om)::value;
#pragma unroll
        for (uint32_t r = 0; r < OM; r++) {
          if (r < O && in) {
            float ay = 0.f;
#pragma unroll
            for (uint32_t k = 0; k < OM; k++)
              if (k < O) ay = fmaf(Ai[r * O + k], y[k], ay);
            quad_y = fmaf(y[r], ay, quad_y);
            lin = fmaf(bi[r], y[r], lin);
            g[r] = 2.f * (ay - bi[r]) / (float)q.B;
          }
        }
      };
      if (O <= 4) outputs(std::integral_constant<uint32_t, 4>{});
      else outputs(std::integral_constant<uint32_t, 16>{});
      uint8_t *d = dy + tid / 8 * rsd + tid % 8 * 16;
      *reinterpret_cast<uint4 *>(d) = make_uint4(pack2(g[0], g[1]), pack2(g[2], g[3]), pack2(g[4], g[5]), pack2(g[6], g[7]));
      *reinterpret_cast<uint4 *>(d + 128) =
          make_uint4(pack2(g[8], g[9]), pack2(g[10], g[11]), pack2(g[12], g[13]), pack2(g[14], g[15]));
      const float ci = stage_abc ? abc[kT * 20 + tid] : (q.c && in ? q.c[row0 + tid] : 0.f);
      float li = in ? (quad_y - 2.f * lin + ci) / (float)q.B : 0.f;
      for (uint32_t r = 0; r <= O; r++) {
        float v = li;
#pragma unroll
        for (uint32_t k = 0; k < 16; k++)
          if (k == r && r < O) v = g[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][r] = v;
      }
    }
    publish();
    if (tid == 0) {
      for (uint32_t t = 0; t < MT; t++) {
        mma_steps(tmem + c_a + t * kT, kmajor(a_w3 + t * 16 * rs3, rs3), kmajor(a_dy, rsd), id_d2, 1);
        mma_steps(tmem + c_w3 + t * 16, kmajor(a_h2 + t * 16 * kH, kH), mnmajor(a_dy, rsd), id_w3, kT / 16);
      }
      tc::mma_commit(&bar);
    }
    if (tid <= O) acc1(tid < O ? s.off[5] + tid : s.n_params, red[0][tid] + red[1][tid]);
    if (!(ok = arrived(&bar, ph))) break;
    const float gb2 = upstream(c_a, h2, m2);  // dz2 takes h2's place
    {
      float v[16];
      tc::tmem_ld16(my + c_w3 + tl * 16, v);
      float *d = slot + s.off[4] + (uint64_t)n * O;
      if (n < W && O == 4 && W % 4 == 0 && !pass) {
        *reinterpret_cast<float4 *>(d) = make_float4(v[0], v[1], v[2], v[3]);
      } else if (n < W) {
#pragma unroll
        for (uint32_t o = 0; o < 16; o++)
          if (o < O) d[o] = pass ? d[o] + v[o] : v[o];
      }
    }
    publish();
    if (tid == 0) {
      for (uint32_t t = 0; t < MT; t++)
        mma_steps(tmem + c_b + t * kT, kmajor(a_w2 + t * 16 * rs2, rs2), mnmajor(a_h2, kH), id_d1, Wp / 16);
      tc::mma_commit(&bar);
      mma_steps(tmem + c_w2, kmajor(a_h2, kH), kmajor(a_h1, kH), id_w2, kT / 16);
      tc::mma_commit(&bar_g);
    }
    if (!(ok = arrived(&bar, ph))) break;
    const float gb1 = upstream(c_b, w2, m1);  // dz1 takes W2's place
    if (n < W) {
      acc1(s.off[1] + n, gb1);
      acc1(s.off[3] + n, gb2);
    }
    publish();
    if (tid == 0) {
      for (uint32_t t = 0; t < MT; t++)
        mma_steps(tmem + c_w1 + t * Ip, kmajor(a_w2 + t * 16 * kH, kH), mnmajor(a_x, rsx), id_w1, kT / 16);
      tc::mma_commit(&bar);
    }
    if (!(ok = arrived(&bar_g, ph_g))) break;
    drain_w2(0);
    if (MT == 2) {
      publish();
      if (tid == 0) {
        mma_steps(tmem + c_w2, kmajor(a_h2 + 16 * kH, kH), kmajor(a_h1, kH), id_w2, kT / 16);
        tc::mma_commit(&bar_g);
      }
    }
    if (!(ok = arrived(&bar, ph))) break;
#pragma unroll 1
    for (uint32_t i0 = 0; i0 < Ip; i0 += 16) {
      float v[16];
      tc::tmem_ld16(my + c_w1 + tl * Ip + i0, v);
      if (n < W)
#pragma unroll
        for (uint32_t j = 0; j < 16; j++)
          if (i0 + j < I) acc1((uint64_t)(i0 + j) * W + n, v[j]);
    }
    if (MT == 2) {
      if (!(ok = arrived(&bar_g, ph_g))) break;
      drain_w2(1);
    }
  }
  if (!ok && tid == 0) {
    if (q.err) atomicOr(q.err, tc::kErrTimeout);
    // copies still in flight land before the CTA exits
    tc::mbar_wait(&wbar1, pass & 1);
    tc::mbar_wait(&wbar2, pass & 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// g[e] = the slots' elements e added in slot order (four contiguous runs of
// slots, then the four sums); element n_params is the loss
__global__ void __launch_bounds__(256) mlp_step_reduce_kernel(const float4 *part, uint32_t slots, uint64_t slot4,
                                                              uint64_t n_params, float *g, float *loss) {
  __shared__ float4 sums[4][64];
  pdl_wait();
  const uint32_t f = threadIdx.x % 64, r = threadIdx.x / 64;
  const uint64_t e4 = (uint64_t)blockIdx.x * 64 + f;
  const uint32_t per = (slots + 3) / 4, k1 = min(slots, (r + 1) * per);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (e4 < slot4)
#pragma unroll 8
    for (uint32_t k = r * per; k < k1; k++) {
      const float4 v = part[k * slot4 + e4];
      a = make_float4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w);
    }
  sums[r][f] = a;
  __syncthreads();
  if (r || e4 >= slot4) return;
  for (uint32_t k = 1; k < 4; k++) {
    const float4 v = sums[k][f];
    a = make_float4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w);
  }
  const float o[4] = {a.x, a.y, a.z, a.w};
  for (uint32_t j = 0; j < 4; j++) {
    const uint64_t e = 4 * e4 + j;
    if (e < n_params) g[e] = o[j];
    else if (e == n_params && loss) *loss = o[j];
  }
}

template <int MT, bool FWD>
cudaError_t launch(const StepParams &q, unsigned grid, cudaStream_t st) {
  const uint32_t Wp = 128 * MT;
  const size_t base = Wp * Wp * 2 + 2 * (size_t)(Wp / 8 * kH) + Wp * 32 + kT * 32 + kT * 21 * 4;
  static std::atomic<uint64_t> configured{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load() & bit)) {
    e = cudaFuncSetAttribute(mlp_step_kernel<MT, FWD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(base + kT * kStepMaxIn * 2));
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit);
  }
  return pdl_launch(mlp_step_kernel<MT, FWD>, grid, 128 * MT, base + kT * q.s.Ip * 2, st, q);
}

}  // namespace

bool mlp_step_shape(uint32_t I, uint32_t W, uint32_t O, const uint64_t off[6], uint64_t n_params, MlpStepShape *s) {
  if (I > kStepMaxIn || W > kStepMaxWidth || O > kStepMaxOut) return false;
  s->I = I;
  s->W = W;
  s->O = O;
  s->Ip = (I + 15) / 16 * 16;
  s->Wp = W <= 128 ? 128 : 256;
  for (int i = 0; i < 6; i++) s->off[i] = off[i];
  s->n_params = n_params;
  s->slot = (n_params + 1 + 3) / 4 * 4;
  return true;
}

cudaError_t mlp_fwd_tc(const MlpStepShape &s, const __nv_bfloat16 *img, const float *params, const float *x,
                       const BlendFeatures &f, uint32_t B, float *y, int *err, cudaStream_t st) {
  StepParams q{s, img, params, x, nullptr, nullptr, nullptr, nullptr, err, B, (B + kT - 1) / kT, f, y};
  const unsigned grid = std::min(q.tiles, kStepSlots);
  return s.Wp == 128 ? launch<1, true>(q, grid, st) : launch<2, true>(q, grid, st);
}

cudaError_t mlp_step(const MlpStepShape &s, const __nv_bfloat16 *img, const float *params, const float *x,
                     const float *A, const float *b, const float *c, uint32_t B, float *part, float *g, float *loss,
                     int *err, cudaStream_t st) {
  StepParams q{s, img, params, x, A, b, c, part, err, B, (B + kT - 1) / kT, {}, nullptr};
  const unsigned grid = std::min(q.tiles, kStepSlots);
  const cudaError_t e = s.Wp == 128 ? launch<1, false>(q, grid, st) : launch<2, false>(q, grid, st);
  if (e != cudaSuccess) return e;
  const uint64_t slot4 = s.slot / 4;
  return pdl_launch(mlp_step_reduce_kernel, (unsigned)((slot4 + 63) / 64), 256, 0, st,
                    reinterpret_cast<const float4 *>(part), grid, slot4, s.n_params, g, loss);
}

}  // namespace mb
