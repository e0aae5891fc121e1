// zf_ldl.cuh -- device parts of the direct zero-forcing solve W = A^{-1} C,
// A = C C^H, by one CTA of 256 threads with C in shared memory: Gram, L D L^H
// with L^{-1}, and the two products (zf.cu in FP32 and FP64, zf_direct.cu for
// the mixed-precision path).
#pragma once
#include "common.cuh"

namespace mb {

template <typename T>
struct Cplx {
  T x, y;
};

template <typename T>
__device__ __forceinline__ Cplx<T> mk(T a, T b) {
  Cplx<T> c;
  c.x = a;
  c.y = b;
  return c;
}

// C[u][b] = csi[b][u] into Cs (leading dimension ldc), coalesced in b K + u
template <typename T>
__device__ __forceinline__ void zf_load_c(const float2 *cg, Cplx<T> *Cs, uint32_t M, uint32_t K, uint32_t ldc) {
  constexpr uint32_t nt = 256;
  const uint32_t tid = threadIdx.x, db = nt / K, du = nt % K;
  uint32_t b = tid / K, u = tid % K;
#pragma unroll 4
  for (uint32_t e = tid; e < M * K; e += nt) {
    const float2 v = cg[e];
    Cs[u * ldc + b] = mk<T>((T)v.x, (T)v.y);
    b += db;
    u += du;
    if (u >= K) {
      u -= K;
      b++;
    }
  }
}

// Gram A = C C^H (both triangles): rows ti + 16 a, columns tj + 16 b of the
// thread, the lower triangle's 16 x 16 blocks.  K <= KP.
template <typename T, int KP>
__device__ __forceinline__ void zf_gram(const Cplx<T> *Cs, Cplx<T> *A, uint32_t M, uint32_t K, uint32_t ldc,
                                        uint32_t lda) {
  using C = Cplx<T>;
  constexpr int GT = KP / 16;
  const uint32_t ti = threadIdx.x / 16, tj = threadIdx.x % 16;
  C acc[GT][GT];
#pragma unroll
  for (int a = 0; a < GT; a++)
#pragma unroll
    for (int b = 0; b < GT; b++) acc[a][b] = mk<T>((T)0, (T)0);
  const C *ca[GT], *cb[GT];
#pragma unroll
  for (int a = 0; a < GT; a++) {
    // rows past K repeat row K - 1: their outputs are not stored
    ca[a] = Cs + min(ti + 16 * a, K - 1) * ldc;
    cb[a] = Cs + min(tj + 16 * a, K - 1) * ldc;
  }
#pragma unroll 4
  for (uint32_t m = 0; m < M; m++) {
    C av[GT], bv[GT];
#pragma unroll
    for (int a = 0; a < GT; a++) {
      av[a] = ca[a][m];
      bv[a] = cb[a][m];
    }
#pragma unroll
    for (int a = 0; a < GT; a++)
#pragma unroll
      for (int b = 0; b <= a; b++) {
        acc[a][b].x += av[a].x * bv[b].x + av[a].y * bv[b].y;
        acc[a][b].y += av[a].y * bv[b].x - av[a].x * bv[b].y;
      }
  }
#pragma unroll
  for (int a = 0; a < GT; a++)
#pragma unroll
    for (int b = 0; b <= a; b++) {
      const uint32_t i = ti + 16 * a, j = tj + 16 * b;
      if (i >= K || j > i) continue;
      const C v = acc[a][b];
      A[i * lda + j] = v;
      if (j < i) A[j * lda + i] = mk<T>(v.x, -v.y);
    }
}

// Rows i > k of the K x K Hermitian A minus a_ik / a_kk times row k, pivot by
// pivot, the multipliers' negatives left in the eliminated entries and taken
// along like the rest of their row: A = L D L^H ends as D on the diagonal and
// L^{-1} strictly below it (what lies above is scratch).  The row of thread t is t / TPR, its
// columns t % TPR + TPR m in registers, rotated by one slot every TPR pivots
// so that the pivot column always sits in slot 0; the pivot row goes through
// shared memory, two buffers of KP at prow (A itself will do, free while the
// rows are in registers; a small A's buffers run on into the 1 KB behind it):
// one barrier a pivot.  *not_pd = 1 when a pivot is not positive.
template <typename T, int KP>
__device__ __forceinline__ void ldl_eliminate(Cplx<T> *A, uint32_t lda, uint32_t K, int *not_pd, Cplx<T> *prow) {
  constexpr int TPR = 256 / KP, NC = KP / TPR > 0 ? KP / TPR : 1;
  const uint32_t i = threadIdx.x / TPR, sub = threadIdx.x % TPR;
  Cplx<T> v[NC];
#pragma unroll
  for (int m = 0; m < NC; m++) {
    const uint32_t c = sub + TPR * m;
    v[m] = i < K && c < K ? A[i * lda + c] : mk<T>(i == c ? (T)1 : (T)0, (T)0);
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t r = 0; r < (uint32_t)NC && r * TPR < K; r++) {
#pragma unroll
    for (int s = 0; s < TPR; s++) {
      const uint32_t k = r * TPR + s;
      if (k < K) {  // uniform
        Cplx<T> f;  // this row's entry in column k
        f.x = __shfl_sync(0xffffffffu, v[0].x, s, TPR);
        f.y = __shfl_sync(0xffffffffu, v[0].y, s, TPR);
        Cplx<T> *pr = prow + (k & 1) * KP;
        if (i == k) {
          T d = f.x;
          if (!(d > (T)0)) {
            *not_pd = 1;
            d = (T)1;
          }
          // in the buffer the pivot's own slot carries 1 / d
          if (sub == (uint32_t)s) v[0] = mk<T>(d, (T)0);
#pragma unroll
          for (int m = 0; m < NC; m++) pr[sub + TPR * m] = v[m];
          if (sub == (uint32_t)s) pr[s] = mk<T>((T)1 / d, (T)0);
        }
        __syncthreads();
        if (i > k) {
          const T inv = pr[s].x;
          const Cplx<T> q = mk<T>(f.x * inv, f.y * inv);
#pragma unroll
          for (int m = 0; m < NC; m++) {
            const Cplx<T> w = pr[sub + TPR * m];
            v[m].x -= q.x * w.x - q.y * w.y;
            v[m].y -= q.x * w.y + q.y * w.x;
          }
          if (sub == (uint32_t)s) v[0] = mk<T>(-q.x, -q.y);
        }
      }
    }
    const Cplx<T> t = v[0];
#pragma unroll
    for (int m = 0; m < NC - 1; m++) v[m] = v[m + 1];
    v[NC - 1] = t;
  }
  __syncthreads();
  // slot m holds column sub + TPR ((m + rotations) % NC)
  const uint32_t rot = min((uint32_t)NC, (K + TPR - 1) / TPR);
  if (i < K) {
#pragma unroll
    for (int m = 0; m < NC; m++) {
      uint32_t c = m + rot;
      if (c >= (uint32_t)NC) c -= NC;
      c = sub + TPR * c;
      if (c <= i) A[i * lda + c] = v[m];
    }
  }
  __syncthreads();
}

// W = L^{-H} D^{-1} (L^{-1} C) in place in Cs, over blocks of four rows: thread
// (part, column b), `cols` columns and `parts` blocks side by side.
// Z = L^{-1} C from the last rows up (a row reads the rows above it), then
// L^{-H} D^{-1} Z from the first rows down; the barriers keep the blocks of one
// round, whose rows read one another's old values, apart.  U steps of a row are
// unrolled.
template <typename T, int U = 4>
__device__ __forceinline__ void ldl_products(const Cplx<T> *A, Cplx<T> *Cs, uint32_t M, uint32_t K, uint32_t ldc,
                                             uint32_t lda) {
  using C = Cplx<T>;
  constexpr uint32_t nt = 256;
  const uint32_t tid = threadIdx.x;
  uint32_t cols = 32;
  while (cols < M && cols < nt) cols *= 2;
  const uint32_t parts = nt / cols, part = tid / cols, nb = (K + 3) / 4;
  for (uint32_t b0 = 0; b0 < M; b0 += cols) {
    const uint32_t b = b0 + tid % cols;
    const bool on = b < M;
    for (uint32_t r = 0; r < nb; r += parts) {
      const uint32_t i0 = r + part < nb ? 4 * (nb - 1 - r - part) : 0;
      const bool act = on && r + part < nb;
      C z[4];
      if (act) {
#pragma unroll
        for (int q = 0; q < 4; q++) z[q] = i0 + q < K ? Cs[(i0 + q) * ldc + b] : mk<T>((T)0, (T)0);
        const C *l[4];
#pragma unroll
        for (int q = 0; q < 4; q++) l[q] = A + min(i0 + q, K - 1) * lda;
#pragma unroll U
        for (uint32_t k = 0; k < i0; k++) {
          const C c = Cs[k * ldc + b];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const C w = l[q][k];
            z[q].x += w.x * c.x - w.y * c.y;
            z[q].y += w.x * c.y + w.y * c.x;
          }
        }
        // within the block: rows i0 .. i0 + 2 of C
#pragma unroll
        for (int k = 0; k < 3; k++) {
          if (i0 + k + 1 >= K) break;
          const C c = Cs[(i0 + k) * ldc + b];
#pragma unroll
          for (int q = k + 1; q < 4; q++) {
            const C w = l[q][i0 + k];
            if (i0 + q < K) {
              z[q].x += w.x * c.x - w.y * c.y;
              z[q].y += w.x * c.y + w.y * c.x;
            }
          }
        }
      }
      if (parts > 1) __syncthreads();
      if (act) {
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (i0 + q < K) {
            const T d = (T)1 / A[(i0 + q) * lda + i0 + q].x;
            Cs[(i0 + q) * ldc + b] = mk<T>(z[q].x * d, z[q].y * d);
          }
      }
      if (parts > 1) __syncthreads();
    }
    for (uint32_t r = 0; r < nb; r += parts) {
      const uint32_t i0 = 4 * (r + part);
      const bool act = on && r + part < nb;
      C z[4];
      if (act) {
#pragma unroll
        for (int q = 0; q < 4; q++) z[q] = i0 + q < K ? Cs[(i0 + q) * ldc + b] : mk<T>((T)0, (T)0);
#pragma unroll
        for (int k = 1; k < 4; k++) {
          if (i0 + k >= K) break;
          const C c = Cs[(i0 + k) * ldc + b];
#pragma unroll
          for (int q = 0; q < k; q++) {
            const C w = A[(i0 + k) * lda + i0 + q];  // conj
            z[q].x += w.x * c.x + w.y * c.y;
            z[q].y += w.x * c.y - w.y * c.x;
          }
        }
#pragma unroll U
        for (uint32_t k = i0 + 4; k < K; k++) {
          const C c = Cs[k * ldc + b];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const C w = A[k * lda + i0 + q];
            z[q].x += w.x * c.x + w.y * c.y;
            z[q].y += w.x * c.y - w.y * c.x;
          }
        }
      }
      if (parts > 1) __syncthreads();
      if (act) {
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (i0 + q < K) Cs[(i0 + q) * ldc + b] = z[q];
      }
      if (parts > 1) __syncthreads();
    }
  }
  __syncthreads();
}

}  // namespace mb
