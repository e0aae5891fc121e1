// zf_direct.cu -- the mixed-precision detector of cells with few users, its
// inverse by a direct FP32 solve.
//
// The tensor-core kernel (zf_mixed.cu) spends a small group on latency: MMA
// round trips, pivots and refinement steps of a few hundred cycles each, two
// CTAs per SM.  With up to 16 users the whole solve on the CUDA cores is
// shorter than those round trips and small enough in registers and shared
// memory for four CTAs per SM: FP32 Gram, its inverse X from L D L^H, and the
// caller's Newton-Schulz steps on one entry a thread.  The rest is
// zf_mixed.cu's: the 1-norm condition estimate, W = X C from BF16 X and C with
// FP32 sums, the BF16 detector image, W (FP32) where asked for, and the FP64
// solve of groups above the threshold or not positive definite in FP32.
// 205 groups: 64 x 16 17 -> 12 us, 128 x 16 23 -> 18 us, 256 x 8 29 -> 16 us
// (launch included); the same solve for 32 users loses (128 x 32: 34 -> 48 us),
// its FP32 products outweigh the round trips.  32 uneven cells, 25 of them with
// K <= 16: 675 -> 605 us a batched slot.
#include <algorithm>
#include <atomic>

#include "eq_tc.cuh"
#include "zf.cuh"
#include "zf_fp64.cuh"
#include "zf_ldl.cuh"

namespace mb {
namespace {

struct ZfdParams {
  float2 *csi;    // [G][M][K]: CSI in, W out
  uint8_t *img;   // [G] detector images
  int32_t *status;
  float *cond, *wmax;
  uint32_t M, K, Mp, MM, nkt;
  uint32_t write_w, ns_iters;
  float cond_thr;
};

// bytes of C, or of the FP64 solve's tile (at least its two pivot buffers)
__host__ __device__ __forceinline__ uint32_t zfd_c_bytes(uint32_t M, uint32_t K) {
  const uint32_t c = (K * (M + 1) * (uint32_t)sizeof(float2) + 15) / 16 * 16, t = zf_fp64_tile_bytes(K);
  return c > t ? c : t > 512 ? t : 512;
}

// the largest of a block's values; red: 8 floats
__device__ __forceinline__ float block_max(float v, float *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();  // red may still be read by the previous call
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = v;
  __syncthreads();
  v = red[0];
#pragma unroll
  for (int w = 1; w < 8; w++) v = fmaxf(v, red[w]);
  return v;
}

__device__ __forceinline__ float2 bf16_round(float2 v) {
  return __bfloat1622float2(__floats2bfloat162_rn(v.x, v.y));
}

// W = X C into Cs in place: thread (part, antenna) forms NB blocks of four
// users; parts = 4 / NB blocks of threads share an antenna's column
template <int NB>
__device__ __forceinline__ void product_bf16(const float2 *Xt, Cplx<float> *Cs, uint32_t M, uint32_t K, uint32_t ldc) {
  constexpr uint32_t cols = 64 * NB, parts = 4 / NB;
  const uint32_t part = threadIdx.x / cols, u0 = part * 4 * NB;
  for (uint32_t b0 = 0; b0 < M; b0 += cols) {
    const uint32_t b = b0 + threadIdx.x % cols;
    float2 w[4 * NB];
#pragma unroll
    for (int i = 0; i < 4 * NB; i++) w[i] = make_float2(0.f, 0.f);
    if (b < M) {
#pragma unroll 4
      for (uint32_t v = 0; v < K; v++) {
        const Cplx<float> cv = Cs[v * ldc + b];
        const float2 c = bf16_round(make_float2(cv.x, cv.y));
        const float4 *x = reinterpret_cast<const float4 *>(Xt + v * 16 + u0);
#pragma unroll
        for (int i = 0; i < 2 * NB; i++) {
          const float4 xx = x[i];
          cfma(w[2 * i], make_float2(xx.x, xx.y), c);
          cfma(w[2 * i + 1], make_float2(xx.z, xx.w), c);
        }
      }
    }
    if (parts > 1) __syncthreads();
    if (b < M) {
#pragma unroll
      for (int i = 0; i < 4 * NB; i++)
        if (u0 + i < K) Cs[(u0 + i) * ldc + b] = mk<float>(w[i].x, w[i].y);
    }
  }
}

__global__ void __launch_bounds__(256, 4) zf_direct_kernel(const ZfdParams q) {
  extern __shared__ __align__(16) unsigned char zd_smem[];
  pdl_wait();
  using C = Cplx<float>;
  constexpr int KP = 16;
  constexpr uint32_t TPR = 256 / KP;  // threads per row of A
  const uint32_t g = blockIdx.x, M = q.M, K = q.K, ldc = M + 1, lda = K + 1, tid = threadIdx.x;
  // C [K][M+1] (or the FP64 solve's tile of it), then room for A [K][K+1] in
  // FP64 (FP32 uses half of it)
  C *Cs = reinterpret_cast<C *>(zd_smem);
  double2 *Ad = reinterpret_cast<double2 *>(zd_smem + zfd_c_bytes(M, K));
  C *A = reinterpret_cast<C *>(Ad);
  __shared__ __align__(16) float2 Xt[KP * KP];  // X transposed, rounded to BF16
  __shared__ float2 Gm[KP * (KP + 1)], Xm[KP * (KP + 1)], Tm[KP * (KP + 1)];  // Newton-Schulz, zero padded
  __shared__ int not_pd;
  __shared__ float red[8];
  float2 *cg = q.csi + (uint64_t)g * M * K;
  uint8_t *img = q.img + (uint64_t)g * q.nkt * q.MM * kZfTile * 2;
  if (tid == 0) not_pd = 0;
  zf_load_c<float>(cg, Cs, M, K, ldc);
  __syncthreads();
  zf_gram<float, KP>(Cs, A, M, K, ldc, lda);
  __syncthreads();
  const uint32_t i = tid / TPR, j = tid % TPR;  // this thread's entry of the K x K matrices
  const bool in = i < K && j < K;
  // largest row sum of |A| (Hermitian: the 1-norm)
  auto norm1 = [&](float2 v) {
    float rs = in ? sqrtf(v.x * v.x + v.y * v.y) : 0.f;
#pragma unroll
    for (uint32_t o = 1; o < TPR; o *= 2) rs += __shfl_xor_sync(0xffffffffu, rs, o);
    return block_max(rs, red);
  };
  const float2 gij = in ? make_float2(A[i * lda + j].x, A[i * lda + j].y) : make_float2(0.f, 0.f);
  const float a1 = norm1(gij);
  ldl_eliminate<float, KP>(A, lda, K, &not_pd, A);
  float cond = INFINITY;
  int st = 2;
  if (!not_pd) {  // uniform
    // X = L^{-H} D^{-1} L^{-1}
    float2 x = make_float2(0.f, 0.f);
    if (in)
      for (uint32_t k = max(i, j); k < K; k++) {
        const C li = k == i ? mk<float>(1.f, 0.f) : A[k * lda + i], lj = k == j ? mk<float>(1.f, 0.f) : A[k * lda + j];
        const float d = 1.f / A[k * lda + k].x;
        x.x = fmaf(li.x * lj.x + li.y * lj.y, d, x.x);
        x.y = fmaf(li.x * lj.y - li.y * lj.x, d, x.y);
      }
    // X <- X (2I - G X)
    const uint32_t o = i * (KP + 1) + j;
    Gm[o] = gij;
    for (uint32_t it = 0; it < q.ns_iters; it++) {
      Xm[o] = x;
      __syncthreads();
      float2 s = make_float2(i == j ? -2.f : 0.f, 0.f);
#pragma unroll
      for (uint32_t k = 0; k < KP; k++) cfma(s, Gm[i * (KP + 1) + k], Xm[k * (KP + 1) + j]);
      Tm[o] = make_float2(-s.x, -s.y);
      __syncthreads();
      x = make_float2(0.f, 0.f);
#pragma unroll
      for (uint32_t k = 0; k < KP; k++) cfma(x, Xm[i * (KP + 1) + k], Tm[k * (KP + 1) + j]);
      __syncthreads();  // the next step overwrites X
    }
    Xt[j * KP + i] = bf16_round(x);
    cond = a1 * norm1(x);  // its barriers also publish Xt
    if (cond <= q.cond_thr) st = 0;
  }
  float mx = 0.f;
  if (st == 0) {
    if (M <= 64) product_bf16<1>(Xt, Cs, M, K, ldc);
    else if (M <= 128) product_bf16<2>(Xt, Cs, M, K, ldc);
    else product_bf16<4>(Xt, Cs, M, K, ldc);
    __syncthreads();
    // the image: user u's rows 2u / 2u + 1 (Re, Im), 8 antennas of both planes
    // an item; antennas past M are zero
    const uint32_t nch = q.Mp / 8, di = 256 / K, du = 256 % K;
    uint32_t ch = tid / K, u = tid % K;
    for (uint32_t e = tid; e < nch * K; e += 256) {
      const C *src = Cs + u * ldc + ch * 8;
      uint32_t re[4], im[4];
#pragma unroll
      for (uint32_t h = 0; h < 4; h++) {
        const C w0 = ch * 8 + 2 * h < M ? src[2 * h] : mk<float>(0.f, 0.f);
        const C w1 = ch * 8 + 2 * h + 1 < M ? src[2 * h + 1] : mk<float>(0.f, 0.f);
        const __nv_bfloat162 r2 = __floats2bfloat162_rn(w0.x, w1.x), i2 = __floats2bfloat162_rn(w0.y, w1.y);
        re[h] = *reinterpret_cast<const uint32_t *>(&r2);
        im[h] = *reinterpret_cast<const uint32_t *>(&i2);
      }
      const uint4 r4 = make_uint4(re[0], re[1], re[2], re[3]), i4 = make_uint4(im[0], im[1], im[2], im[3]);
      *reinterpret_cast<uint4 *>(img + img_off(2 * u, ch * 8, q.MM)) = r4;
      *reinterpret_cast<uint4 *>(img + img_off(2 * u + 1, ch * 8, q.MM)) = i4;
      *reinterpret_cast<uint4 *>(img + img_off(2 * u, q.Mp + ch * 8, q.MM)) =
          make_uint4(i4.x ^ 0x80008000u, i4.y ^ 0x80008000u, i4.z ^ 0x80008000u, i4.w ^ 0x80008000u);
      *reinterpret_cast<uint4 *>(img + img_off(2 * u + 1, q.Mp + ch * 8, q.MM)) = r4;
      ch += di;
      u += du;
      if (u >= K) {
        u -= K;
        ch++;
      }
    }
    if (q.write_w) {
      uint32_t b = tid / K, v = tid % K;
#pragma unroll 4
      for (uint32_t e = tid; e < M * K; e += 256) {
        const C w = Cs[v * ldc + b];
        cg[e] = make_float2(w.x, w.y);
        mx = fmaxf(mx, sqrtf(w.x * w.x + w.y * w.y));
        b += di;
        v += du;
        if (v >= K) {
          v -= K;
          b++;
        }
      }
    }
  } else {
    // half as many antennas in FP64 as C has in FP32, an odd number
    const uint32_t T = max(kFp64Tile, ((M + 1) / 2 - 1) | 1u);
    const Fp64Group r = zf_fp64_group_call<KP, 64>(cg, img, Ad, reinterpret_cast<double2 *>(Cs), T, &not_pd, M, K);
    st = r.status;
    mx = r.wmax;
  }
  if (q.wmax) {
    mx = block_max(mx, red);
    if (tid == 0) q.wmax[g] = mx;
  }
  if (tid == 0) {
    if (q.status) q.status[g] = st;
    if (q.cond) q.cond[g] = cond;
  }
}

size_t zfd_smem(uint32_t M, uint32_t K) {
  // the pivot buffers of a small A reach past it (two of 16 entries)
  return zfd_c_bytes(M, K) + std::max<size_t>((size_t)K * (K + 1) * sizeof(double2), 2 * 16 * sizeof(float2));
}

}  // namespace

mb_status zf_direct_run(float2 *csi, void *img, uint32_t groups, uint32_t M, uint32_t K, uint32_t ns_iters,
                        float cond_thr, int32_t *status, float *cond, cudaStream_t st, bool write_w, float *wmax) {
  const TcShape s = tc_shape(M, K);
  const ZfdParams p{csi, reinterpret_cast<uint8_t *>(img), status, cond, write_w ? wmax : nullptr, M, K, s.Mp, s.MM,
                    s.nkt, write_w ? 1u : 0u, ns_iters, cond_thr};
  const size_t smem = zfd_smem(M, K);
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> limit{0};
  int dev = 0, maxs = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load() & bit)) {
    MB_CUDA_TRY(cudaDeviceGetAttribute(&maxs, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa;
    MB_CUDA_TRY(cudaFuncGetAttributes(&fa, zf_direct_kernel));
    MB_CUDA_TRY(cudaFuncSetAttribute(zf_direct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     maxs - (int)fa.sharedSizeBytes));
    limit = maxs - (int)fa.sharedSizeBytes;
    configured.fetch_or(bit);
  }
  if (K > 16 || smem > (size_t)limit.load()) return MB_UNSUPPORTED;
  if (groups == 0) return MB_OK;
  MB_CUDA_TRY(pdl_launch(zf_direct_kernel, groups, 256, smem, st, p));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

}  // namespace mb
