// gj.cuh -- Gauss-Jordan inverse of a small Hermitian matrix by one CTA,
// shared by the mixed-precision ZF and the per-subcarrier detector.
#pragma once
#include "common.cuh"

namespace mb {

// Inverse of the K x K Hermitian positive definite matrix G (leading dim ld)
// into X by in-place Gauss-Jordan without pivoting (every pivot of a
// positive definite matrix is real and positive): at pivot k the pivot row
// becomes a_kj / a_kk with a_kk <- 1 / a_kk, and every other row i becomes
// a_ij - a_ik a_kj' with a_ik <- -a_ik / a_kk, so column k of G is replaced
// by column k of the inverse and no identity half is carried.  The matrix is
// padded to KP x KP with an identity block.  Thread t holds row t / TPR in
// registers, columns t % TPR + TPR m; the pivot row goes through shared
// memory (prow, two buffers of KP), so each pivot costs one barrier.  The
// register row is rotated by one slot after every TPR pivots, so the pivot
// column always sits in slot 0 and the loop body indexes registers
// statically without being unrolled over the row (a short body: the
// unrolled form stalled on instruction fetch at KP = 64).
// 256 threads; X may be G; *bad must be 0 (before a barrier).  Returns false
// when a pivot is not positive (the output is then garbage).
template <int KP>
__device__ __forceinline__ bool gj_inverse(const float2 *G, float2 *X, uint32_t K, uint32_t ld,
                                           float2 *prow, int *bad) {
  constexpr int TPR = 256 / KP, NC = KP / TPR;
  const uint32_t i = threadIdx.x / TPR, sub = threadIdx.x % TPR;
  // v[m] holds column sub + TPR ((m + r) % NC) after r rotations
  float2 v[NC];
#pragma unroll
  for (int m = 0; m < NC; m++) {
    const uint32_t c = sub + TPR * m;
    v[m] = (i < K && c < K) ? G[i * ld + c] : make_float2(i == c ? 1.f : 0.f, 0.f);
  }
#pragma unroll 1
  for (uint32_t r = 0; r < (uint32_t)NC; r++) {
#pragma unroll
    for (int s = 0; s < TPR; s++) {
      const uint32_t k = r * TPR + s;
      float2 f;  // this row's entry in column k
      f.x = __shfl_sync(0xffffffffu, v[0].x, s, TPR);
      f.y = __shfl_sync(0xffffffffu, v[0].y, s, TPR);
      float2 *pr = prow + (k & 1) * KP;
      if (i == k) {
        if (!(f.x > 0.f)) *bad = 1;
        const float inv = __frcp_rn(f.x);
        if (sub == (uint32_t)s) v[0] = make_float2(1.f, 0.f);
#pragma unroll
        for (int m = 0; m < NC; m++) {
          v[m].x *= inv;
          v[m].y *= inv;
          pr[sub + TPR * m] = v[m];
        }
      }
      __syncthreads();
      if (i != k) {
        if (sub == (uint32_t)s) v[0] = make_float2(0.f, 0.f);
#pragma unroll
        for (int m = 0; m < NC; m++) {
          const float2 w = pr[sub + TPR * m];
          v[m].x -= f.x * w.x - f.y * w.y;
          v[m].y -= f.x * w.y + f.y * w.x;
        }
      }
    }
    const float2 t = v[0];
#pragma unroll
    for (int m = 0; m < NC - 1; m++) v[m] = v[m + 1];
    v[NC - 1] = t;
  }
  __syncthreads();
  const bool ok = *bad == 0;
  if (i < K) {
#pragma unroll
    for (int m = 0; m < NC; m++) {
      const uint32_t c = sub + TPR * m;
      if (c < K) X[i * ld + c] = v[m];
    }
  }
  __syncthreads();
  return ok;
}

}  // namespace mb
