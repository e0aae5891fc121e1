// zf.cu -- per-subcarrier-group zero-forcing detector and precoder.
//
// Replaces Beamform::beamformer_uplink (beamform/beamform.cu:74-122: cuBLAS
// CgemmStridedBatched for the Gram C C^H, cusolverDnCpotrfBatched and
// cusolverDnCpotrsBatched with G*M single right-hand sides) with ONE CTA per
// subcarrier group that keeps C in shared memory for the whole solve: Gram,
// L D L^H (Cholesky without the square roots) with L^{-1}, the products of
// W = (C C^H)^{-1} C with it and the write-back in the CSI layout.  The downlink precoder P = W^T / max|W|
// (beam_utils.cuh:40-80) can be emitted from the same CTA.
//
// FP32 (MB_ZF_FP32) has the reference's precision; FP64 (MB_ZF_FP64)
// runs the same schedule in double.  Unlike the reference, which ignores
// cuSOLVER's info array, a non positive definite Gram is reported per group
// (status 1) and its W is zeroed.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "zf.cuh"
#include "zf_ldl.cuh"

namespace mb {

// Fills the missing users of a short last group from group G-2 (see
// mb_zf_uplink); runs before the solve so the in-place update of group G-2
// cannot race with the read.
__global__ void zf_fill_tail_kernel(float2 *csi, uint32_t G, uint32_t M,
                                    uint32_t K, uint32_t rem, uint32_t sg) {
  pdl_wait();
  const uint64_t total = (uint64_t)M * K;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
       e += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t u = (uint32_t)(e % K);
    if ((u % sg) >= rem) {
      csi[(uint64_t)(G - 1) * total + e] = csi[(uint64_t)(G - 2) * total + e];
    }
  }
}

// One CTA per group.  Shared memory: C as [K][M+1] complex of T, A as
// [K][K+1].  W = A^{-1} C as L^{-H} D^{-1} (L^{-1} C): with L^{-1} at hand both
// products run over all rows and antennas at once, where the triangular
// solves of a Cholesky factor left one thread per antenna a chain of K^2
// dependent steps and the factor itself three barriers a column.  Latency
// bound for small cells (75 groups of 64 x 16: 20.4 us
// before, 9.0 us).
// KP: users the elimination has registers for, KG: the Gram's blocks of 16
// (three instead of four from 33 to 48 users, in FP32: 205 groups of 256 x 33
// 102.5 -> 85 us, of 256 x 48 174 -> 153; the Cholesky form 96 and 266).
template <typename T, int KP, int KG>
__global__ void __launch_bounds__(256)
    zf_chol_kernel(float2 *csi, float2 *precoder, uint32_t M, uint32_t K,
                   int32_t *status, float *cond_out) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char zf_smem_raw[];
  using C = Cplx<T>;
  const uint32_t g = blockIdx.x;
  const uint32_t ldc = M + 1, lda = K + 1;
  C *Cs = reinterpret_cast<C *>(zf_smem_raw);
  C *A = Cs + (size_t)K * ldc;
  float *red = reinterpret_cast<float *>(A + (size_t)K * lda);
  __shared__ int not_pd;
  const uint32_t tid = threadIdx.x;
  constexpr uint32_t nt = 256;
  float2 *cg = csi + (uint64_t)g * M * K;

  if (tid == 0) not_pd = 0;
  const uint32_t db = nt / K, du = nt % K;
  zf_load_c<T>(cg, Cs, M, K, ldc);
  __syncthreads();
  zf_gram<T, KG>(Cs, A, M, K, ldc, lda);
  __syncthreads();
  ldl_eliminate<T, KP>(A, lda, K, &not_pd, A);
  const bool bad = not_pd != 0;
  ldl_products<T>(A, Cs, M, K, ldc, lda);

  // write W back in the CSI layout; track max |W| for the precoder
  float mx = 0.f;
  {
    uint32_t b = tid / K, u = tid % K;
#pragma unroll 4
    for (uint32_t e = tid; e < M * K; e += nt) {
      const C w = Cs[u * ldc + b];
      const float2 o = bad ? make_float2(0.f, 0.f) : make_float2((float)w.x, (float)w.y);
      cg[e] = o;
      mx = fmaxf(mx, sqrtf(o.x * o.x + o.y * o.y));
      b += db;
      u += du;
      if (u >= K) {
        u -= K;
        b++;
      }
    }
  }
  if (status && tid == 0) status[g] = bad ? 1 : 0;
  if (cond_out && tid == 0) {
    // cheap estimate from the pivots: max d_ii / min d_ii
    T lo = A[0].x, hi = A[0].x;
    for (uint32_t i = 1; i < K; i++) {
      T d = A[i * lda + i].x;
      lo = d < lo ? d : lo;
      hi = d > hi ? d : hi;
    }
    cond_out[g] = bad ? INFINITY : (float)(hi / lo);
  }
  if (!precoder) return;
  red[tid] = mx;
  __syncthreads();
  for (uint32_t s = nt / 2; s > 0; s >>= 1) {
    if (tid < s) red[tid] = fmaxf(red[tid], red[tid + s]);
    __syncthreads();
  }
  const float inv = 1.0f / red[0];
  float2 *pg = precoder + (uint64_t)g * M * K;
  for (uint32_t u = tid / 32; u < K; u += nt / 32)
    for (uint32_t b = tid % 32; b < M; b += 32) {
      const C w = Cs[u * ldc + b];
      const float2 o = bad ? make_float2(0.f, 0.f) : make_float2((float)w.x, (float)w.y);
      pg[(uint64_t)u * M + b] = make_float2(o.x * inv, o.y * inv);
    }
}

// beam_utils.cuh:40-80 as a standalone kernel: a cluster of CTAs per group,
// each with mb antennas of it in shared memory.  W is read once (a CTA per
// group that read it for the maximum and again, tile by tile between
// barriers, for the transposition took 38 us for 205 groups of 256 x 64;
// 16 us here); the group's maximum crosses the cluster through
// distributed shared memory.  HBM bound: W in, P out.
__global__ void __launch_bounds__(256)
    precoder_kernel(const float2 *W, float2 *P, uint32_t M, uint32_t K, uint32_t mb) {
  namespace cg = cooperative_groups;
  extern __shared__ float2 pc_tile[];  // [mb][ldt]
  pdl_wait();
  __shared__ float red[8], cmax;
  const cg::cluster_group cl = cg::this_cluster();
  const uint32_t cn = cl.num_blocks(), rank = cl.block_rank(), g = blockIdx.x / cn;
  const uint32_t b0 = rank * mb, nb = b0 < M ? min(mb, M - b0) : 0, ldt = K | 1;
  const uint32_t lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const float2 *wg = W + ((uint64_t)g * M + b0) * K;
  float mx = 0.f;
  uint32_t b = threadIdx.x / K, u = threadIdx.x % K;  // element threadIdx.x, then 256 further each time
  const uint32_t db = 256 / K, du = 256 % K;
#pragma unroll 8
  for (uint32_t e = threadIdx.x; e < nb * K; e += 256) {
    const float2 v = wg[e];
    mx = fmaxf(mx, sqrtf(v.x * v.x + v.y * v.y));
    pc_tile[b * ldt + u] = v;
    b += db;
    u += du;
    if (u >= K) {
      u -= K;
      b++;
    }
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) mx = fmaxf(mx, red[w]);
    cmax = mx;
  }
  cl.sync();
  mx = 0.f;
  for (uint32_t r = 0; r < cn; r++) mx = fmaxf(mx, *cl.map_shared_rank(&cmax, r));
  cl.sync();  // no CTA exits while another reads its maximum
  const float inv = 1.0f / mx;
  float2 *pg = P + (uint64_t)g * M * K + b0;
  for (uint32_t r = warp; r < K; r += 8)
    for (uint32_t c = lane; c < nb; c += 32) {
      const float2 v = pc_tile[c * ldt + r];
      pg[(uint64_t)r * M + c] = make_float2(v.x * inv, v.y * inv);
    }
}

// The same for matrices whose eighth exceeds one SM's shared memory (more than
// about 28,000 entries): one CTA per group, W read twice.
__global__ void __launch_bounds__(256)
    precoder_wide_kernel(const float2 *W, float2 *P, uint32_t M, uint32_t K) {
  __shared__ float red[256];
  const uint32_t g = blockIdx.x;
  const float2 *wg = W + (uint64_t)g * M * K;
  float2 *pg = P + (uint64_t)g * M * K;
  float mx = 0.f;
  for (uint32_t e = threadIdx.x; e < M * K; e += blockDim.x) {
    float2 v = wg[e];
    mx = fmaxf(mx, sqrtf(v.x * v.x + v.y * v.y));
  }
  red[threadIdx.x] = mx;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  const float inv = 1.0f / red[0];
  // P[u][b] = W[b][u] * inv through 32 x 32 shared-memory tiles, so both the
  // reads (along u) and the writes (along b) are coalesced
  __shared__ float2 tile[32][33];
  const uint32_t tx = threadIdx.x % 32, ty = threadIdx.x / 32;  // 8 rows of 32
  for (uint32_t b0 = 0; b0 < M; b0 += 32)
    for (uint32_t u0 = 0; u0 < K; u0 += 32) {
      __syncthreads();
      for (uint32_t r = ty; r < 32; r += 8) {
        const uint32_t b = b0 + r, u = u0 + tx;
        tile[r][tx] = (b < M && u < K) ? wg[(uint64_t)b * K + u] : make_float2(0.f, 0.f);
      }
      __syncthreads();
      for (uint32_t r = ty; r < 32; r += 8) {
        const uint32_t u = u0 + r, b = b0 + tx;
        if (u < K && b < M) {
          const float2 v = tile[tx][r];
          pg[(uint64_t)u * M + b] = make_float2(v.x * inv, v.y * inv);
        }
      }
    }
}

// P[g][u][b] = W[g][b][u] / wmax[g]: one CTA per (group, 32 x 32 tile),
// transposed through shared memory
__global__ void __launch_bounds__(256)
    precoder_scale_kernel(const float2 *W, float2 *P, const float *wmax, uint32_t M, uint32_t K,
                          uint32_t tiles_b) {
  __shared__ float2 tile[32][33];
  pdl_wait();
  const uint32_t g = blockIdx.x;
  const uint32_t b0 = (blockIdx.y % tiles_b) * 32, u0 = (blockIdx.y / tiles_b) * 32;
  const uint32_t tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  const float2 *wg = W + (uint64_t)g * M * K;
  float2 *pg = P + (uint64_t)g * M * K;
  const float inv = 1.0f / wmax[g];  // as precoder_kernel
  for (uint32_t r = ty; r < 32; r += 8) {
    const uint32_t b = b0 + r, u = u0 + tx;
    tile[r][tx] = (b < M && u < K) ? wg[(uint64_t)b * K + u] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  for (uint32_t r = ty; r < 32; r += 8) {
    const uint32_t u = u0 + r, b = b0 + tx;
    if (u < K && b < M) {
      const float2 v = tile[tx][r];
      pg[(uint64_t)u * M + b] = make_float2(v.x * inv, v.y * inv);
    }
  }
}

size_t zf_chol_smem(uint32_t M, uint32_t K, bool dbl) {
  size_t c = dbl ? 16 : 8;
  return c * ((size_t)K * (M + 1) + (size_t)K * (K + 1)) + 256 * sizeof(float);
}

mb_status zf_fill_tail(float2 *csi, uint32_t groups, uint32_t S, uint32_t sg,
                       uint32_t M, uint32_t K, cudaStream_t st) {
  if (groups < 2) return MB_OK;
  uint64_t full = (uint64_t)(groups - 1) * sg;
  if (S <= full || S - full >= sg) return MB_OK;
  uint32_t rem = (uint32_t)(S - full);
  uint64_t total = (uint64_t)M * K;
  unsigned blocks = (unsigned)std::min<uint64_t>((total + 255) / 256, 1024);
  MB_CUDA_TRY(pdl_launch(zf_fill_tail_kernel, blocks, 256, 0, st, csi, groups, M, K, rem, sg));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

template <typename T, int KP, int KG = KP>
static mb_status zf_chol_launch(float2 *csi, float2 *precoder, uint32_t groups, uint32_t M, uint32_t K, size_t smem,
                                int32_t *status, float *cond, cudaStream_t st) {
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> static_smem{0};
  int dev = 0, maxs = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  MB_CUDA_TRY(cudaDeviceGetAttribute(&maxs, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load() & bit)) {
    cudaFuncAttributes fa;
    MB_CUDA_TRY(cudaFuncGetAttributes(&fa, zf_chol_kernel<T, KP, KG>));
    MB_CUDA_TRY(cudaFuncSetAttribute(zf_chol_kernel<T, KP, KG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     maxs - (int)fa.sharedSizeBytes));
    static_smem = (int)fa.sharedSizeBytes;
    configured.fetch_or(bit);
  }
  if (smem + (size_t)static_smem.load() > (size_t)maxs) return MB_UNSUPPORTED;
  if (groups == 0) return MB_OK;
  MB_CUDA_TRY(pdl_launch(zf_chol_kernel<T, KP, KG>, groups, 256, smem, st, csi, precoder, M, K, status, cond));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

mb_status zf_chol(float2 *csi, float2 *precoder, uint32_t groups, uint32_t M,
                  uint32_t K, bool dbl, int32_t *status, float *cond,
                  cudaStream_t st) {
  const size_t smem = zf_chol_smem(M, K, dbl);
  if (dbl) {
    auto f = K <= 16   ? zf_chol_launch<double, 16>
             : K <= 32 ? zf_chol_launch<double, 32>
             : K <= 48 ? zf_chol_launch<double, 64, 48>
                       : zf_chol_launch<double, 64>;
    return f(csi, precoder, groups, M, K, smem, status, cond, st);
  }
  auto f = K <= 16   ? zf_chol_launch<float, 16>
           : K <= 32 ? zf_chol_launch<float, 32>
           : K <= 48 ? zf_chol_launch<float, 64, 48>
                     : zf_chol_launch<float, 64>;
  return f(csi, precoder, groups, M, K, smem, status, cond, st);
}

mb_status precoder_scale(const float2 *W, float2 *P, const float *wmax, uint32_t M, uint32_t K,
                         uint32_t groups, cudaStream_t st) {
  if (groups == 0) return MB_OK;
  const uint32_t tb = (M + 31) / 32, tu = (K + 31) / 32;
  MB_CUDA_TRY(pdl_launch(precoder_scale_kernel, dim3(groups, tb * tu), 256, 0, st, W, P, wmax, M, K, tb));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

mb_status precoder_launch(const float2 *W, float2 *P, uint32_t M, uint32_t K,
                          uint32_t groups, cudaStream_t st) {
  if (groups == 0) return MB_OK;
  // 32 antennas a CTA while the portable cluster of eight lasts, more beyond
  uint32_t cn = 1;
  while (cn < 8 && cn * 32 < M) cn *= 2;
  const uint32_t mb = std::max<uint32_t>(32, (M + cn - 1) / cn);
  const size_t smem = sizeof(float2) * (size_t)std::min(mb, M) * (K | 1);
  int dev = 0, maxs = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  MB_CUDA_TRY(cudaDeviceGetAttribute(&maxs, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  if (smem + 1024 > (size_t)maxs || (uint64_t)groups * cn > 0x7FFFFFFFull) {
    // an eighth of W does not fit one SM: two passes over it
    precoder_wide_kernel<<<groups, 256, 0, st>>>(W, P, M, K);
    MB_LAUNCH_CHECK();
    return MB_OK;
  }
  static std::atomic<uint64_t> configured{0};
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load() & bit)) {
    MB_CUDA_TRY(cudaFuncSetAttribute(precoder_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, maxs - 1024));
    configured.fetch_or(bit);
  }
  cudaLaunchAttribute at[2]{};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cn;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as pdl_launch()
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(groups * cn);
  lc.blockDim = dim3(256);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  lc.attrs = at;
  lc.numAttrs = 2;
  MB_CUDA_TRY(cudaLaunchKernelEx(&lc, precoder_kernel, W, P, M, K, mb));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

}  // namespace mb

using namespace mb;

struct mb_zf {
  uint32_t M, K, max_groups;
  void *img_w;        // mixed-precision detector images, sized for max_groups
  const mb_mlp *net;  // network of the learned initial iterate (not owned), or null
};

extern "C" mb_status mb_zf_create(uint32_t num_bs, uint32_t num_ue,
                                  uint32_t max_groups, mb_zf **out) {
  if (!out) return MB_BAD_ARG;
  *out = nullptr;
  if (num_bs == 0 || num_ue == 0 || num_ue > num_bs || num_ue > 64)
    return MB_BAD_SHAPE;
  if (!device_tables()) return MB_CUDA_ERROR;
  mb_zf *z = new mb_zf{num_bs, num_ue, max_groups, nullptr, nullptr};
  const uint64_t bytes = zf_mixed_scratch_bytes(max_groups, num_bs, num_ue);
  cudaError_t e = cudaSuccess;
  if (bytes) e = cudaMalloc(&z->img_w, bytes);
  if (e != cudaSuccess) {
    cudaFree(z->img_w);
    delete z;
    return record_error(e);
  }
  *out = z;
  return MB_OK;
}

extern "C" mb_status mb_zf_destroy(mb_zf *z) {
  if (!z) return MB_BAD_ARG;
  cudaFree(z->img_w);
  delete z;
  return MB_OK;
}

extern "C" mb_status mb_zf_uplink(mb_zf *z, mb_c32 *csi, uint32_t groups,
                                  uint32_t S, uint32_t sg,
                                  const mb_zf_opts *opts, int32_t *status,
                                  float *cond, void *stream) {
  if (!z || !csi) return MB_BAD_ARG;
  if (groups > z->max_groups) return MB_BAD_SHAPE;  // beamform.cu:144-152
  if (sg == 0 || (uint64_t)groups * sg < S || (uint64_t)(groups - 1) * sg >= S)
    return MB_BAD_SHAPE;
  uint32_t prec = opts ? opts->precision : MB_ZF_FP32;
  cudaStream_t st = as_stream(stream);
  float2 *c = reinterpret_cast<float2 *>(csi);
  mb_status s = zf_fill_tail(c, groups, S, sg, z->M, z->K, st);
  if (s != MB_OK) return s;
  switch (prec) {
    case MB_ZF_FP32:
      return zf_chol(c, nullptr, groups, z->M, z->K, false, status, cond, st);
    case MB_ZF_FP64:
      return zf_chol(c, nullptr, groups, z->M, z->K, true, status, cond, st);
    case MB_ZF_MIXED: {
      ZfNetView v{};
      if (opts && opts->init == 1) {
        if (!z->net) return MB_BAD_ARG;
        const mb_status r = mlp_zf_init_view(z->net, &v);
        if (r != MB_OK) return r;
      }
      return zf_mixed_run(c, z->img_w, groups, z->M, z->K, opts, status, cond, st, true, nullptr, &v);
    }
  }
  return MB_BAD_ARG;
}

extern "C" mb_status mb_zf_set_init_net(mb_zf *z, const mb_mlp *net) {
  if (!z) return MB_BAD_ARG;
  if (net) {
    ZfNetView v;
    const mb_status r = mlp_zf_init_view(net, &v);
    if (r != MB_OK) return r;
  }
  z->net = net;
  return MB_OK;
}

extern "C" mb_status mb_zf_precoder(const mb_c32 *W, mb_c32 *P, uint32_t M,
                                    uint32_t K, uint32_t groups, void *stream) {
  if (!W || !P || M == 0 || K == 0) return MB_BAD_ARG;
  return precoder_launch(reinterpret_cast<const float2 *>(W),
                         reinterpret_cast<float2 *>(P), M, K, groups,
                         as_stream(stream));
}
