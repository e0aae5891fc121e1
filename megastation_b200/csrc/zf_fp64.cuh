// zf_fp64.cuh -- the FP64 solve of one group, the fallback of both
// mixed-precision detector kernels (zf_mixed.cu, zf_direct.cu), and the
// detector image's layout.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace mb {

constexpr uint32_t kZfTile = 64;  // antennas per k tile of the image

__device__ __forceinline__ uint32_t img_off(uint32_t r, uint32_t kk, uint32_t MM) {
  // canonical K-major, no swizzle: [k tile][row group][k chunk][row][8]
  const uint32_t kt = kk / kZfTile, kin = kk % kZfTile;
  return kt * (MM * kZfTile * 2) + (r / 8) * 1024 + (kin / 8) * 128 + (r % 8) * 16 + (kin % 8) * 2;
}

// In-place Cholesky of the K x K Hermitian matrix A (lower, leading dim lda)
// by all threads; returns false when a pivot is not positive.
template <typename C, typename R>
__device__ bool chol_smem(C *A, uint32_t K, uint32_t lda, int *flag) {
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) *flag = 0;
  __syncthreads();
  for (uint32_t j = 0; j < K; j++) {
    if (tid == 0) {
      R d = A[j * lda + j].x;
      if (!(d > (R)0)) {
        *flag = 1;
        d = (R)1;
      }
      A[j * lda + j].x = sqrt(d);
      A[j * lda + j].y = 0;
    }
    __syncthreads();
    const R inv = (R)1 / A[j * lda + j].x;
    for (uint32_t i = j + 1 + tid; i < K; i += nt) {
      A[i * lda + j].x *= inv;
      A[i * lda + j].y *= inv;
    }
    __syncthreads();
    const uint32_t rem = K - j - 1;
    for (uint32_t q = tid; q < rem * rem; q += nt) {
      const uint32_t i = j + 1 + q / rem, k = j + 1 + q % rem;
      if (k > i) continue;
      const C a = A[i * lda + j], b = A[k * lda + j];
      A[i * lda + k].x -= a.x * b.x + a.y * b.y;
      A[i * lda + k].y -= a.y * b.x - a.x * b.y;
    }
    __syncthreads();
  }
  return *flag == 0;
}

// Group of cg [M][K] in FP64 (Gram, Cholesky, solve) by all threads: W (FP32)
// over cg, the detector image imgw (MM rows, nkt k tiles), and mx = max(mx,
// |W| of the values this thread stored).  Gd: [K][K+1], *flag scratch, both in
// shared memory; K <= ZMAX.  Returns the group's status: 2, or 1 (not positive
// definite, W zero).
template <int ZMAX>
__device__ __noinline__ int zf_fp64_group(float2 *cg, uint8_t *imgw, double2 *Gd, int *flag, uint32_t M, uint32_t K, uint32_t Mp,
                             uint32_t MM, uint32_t nkt, float &wmx) {
  const uint32_t tid = threadIdx.x, nt = blockDim.x;
  using D2 = double2;
  const uint32_t ldd = K + 1;
  for (uint32_t e = tid; e < K * K; e += nt) {
    const uint32_t i = e / K, j = e % K;
    if (j > i) continue;
    double sr = 0, si = 0;
    for (uint32_t b = 0; b < M; b++) {
      const float2 a = cg[b * K + i], c = cg[b * K + j];
      sr += (double)a.x * c.x + (double)a.y * c.y;
      si += (double)a.y * c.x - (double)a.x * c.y;
    }
    Gd[i * ldd + j] = make_double2(sr, si);
  }
  __syncthreads();
  const bool pd = chol_smem<D2, double>(Gd, K, ldd, flag);
  for (uint32_t c = tid; c < nkt * MM * kZfTile * 2 / 16; c += nt)
    reinterpret_cast<uint4 *>(imgw)[c] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (uint32_t b = tid; b < M; b += nt) {
    D2 z[ZMAX];
    for (uint32_t i = 0; i < K; i++) {
      const float2 cv = cg[b * K + i];
      D2 s = make_double2(cv.x, cv.y);
      for (uint32_t k = 0; k < i && pd; k++) {
        const D2 l = Gd[i * ldd + k];
        s.x -= l.x * z[k].x - l.y * z[k].y;
        s.y -= l.x * z[k].y + l.y * z[k].x;
      }
      const double d = pd ? Gd[i * ldd + i].x : 1.0;
      z[i] = make_double2(s.x / d, s.y / d);
    }
    for (int i = (int)K - 1; i >= 0 && pd; i--) {
      D2 s = z[i];
      for (uint32_t k = i + 1; k < K; k++) {
        const D2 l = Gd[k * ldd + i];
        s.x -= l.x * z[k].x + l.y * z[k].y;
        s.y -= l.x * z[k].y - l.y * z[k].x;
      }
      const double d = Gd[i * ldd + i].x;
      z[i] = make_double2(s.x / d, s.y / d);
    }
    // every thread reads its own column b of C before overwriting it
    for (uint32_t u = 0; u < K; u++) {
      const float2 w = pd ? make_float2((float)z[u].x, (float)z[u].y) : make_float2(0.f, 0.f);
      cg[b * K + u] = w;
      wmx = fmaxf(wmx, sqrtf(w.x * w.x + w.y * w.y));
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u, b, MM)) = __float2bfloat16_rn(w.x);
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u, Mp + b, MM)) = __float2bfloat16_rn(-w.y);
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u + 1, b, MM)) = __float2bfloat16_rn(w.y);
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u + 1, Mp + b, MM)) = __float2bfloat16_rn(w.x);
    }
  }
  return pd ? 2 : 1;
}

}  // namespace mb
