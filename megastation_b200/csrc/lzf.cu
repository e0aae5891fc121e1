// lzf.cu -- per-subcarrier zero forcing with a learned initial iterate.
//
// The reference computes one ZF detector per group of sg subcarriers from
// the comb pilots (beamform/beamform.cu:74-122), which loses accuracy when
// the channel changes within a group (large delay spread).  This module
// builds a detector per subcarrier instead, without a full inversion per
// subcarrier (no counterpart in the reference):
//  1. interpolate each user's comb-pilot estimates linearly along frequency
//     (user u's pilot of group g sits on subcarrier g sg + u mod sg) to a
//     CSI estimate c_s [M][K] for every data subcarrier s (the pilot FFT's
//     CSI convention: the conjugate channel);
//  2. per subcarrier Gram G_s = C C^H with C[u][b] = c_s[b][u], the
//     reference's Gram (FP32; FP64 for training targets);
//  3. exact inverses X_g of the Grams at the group centres only (Gauss-Jordan
//     per matrix);
//  4. an initial iterate per subcarrier X0_s = sum_j alpha_j X_{g+j},
//     j = -1..2 (group indices clamped at the band edges), where alpha comes
//     from the MLP (mlp.cu) evaluated on features of the neighbouring centre
//     Grams and the subcarrier's offset in its group ("learned"), or alpha =
//     (0, 1, 0, 0) ("coarse": the group's own inverse, i.e. the per-group
//     ZF), or X0_s = G_s^{-1} ("exact");
//  5. ns_iters Newton-Schulz steps X <- X (2I - G_s X) per subcarrier;
//  6. the detector W_s = X_s C, stored [S][M][K] like the per-group W with
//     sg = 1, so the existing equalizer applies it unchanged.
// Training targets come from the same interpolation in FP64: with Y_j the
// four centre inverses and X* = G_s^{-1} (FP64), the loss of a blend alpha
// is ||sum_j alpha_j Y_j - X*||_F^2 / ||X*||_F^2 = alpha^T A alpha - 2 b^T
// alpha + 1 with A_jk = Re tr(Y_j^H Y_k) / ||X*||^2, b_j = Re tr(Y_j^H X*) /
// ||X*||^2.
#include <algorithm>
#include <atomic>
#include <vector>

#include "common.cuh"
#include "gj.cuh"
#include "mlp_step.cuh"

namespace mb {
namespace {

constexpr int kBlend = 4;  // centre inverses g-1, g, g+1, g+2

template <typename T> struct CT { using V = float2; };
template <> struct CT<double> { using V = double2; };

template <typename V> __device__ __forceinline__ V cz() { V r; r.x = 0; r.y = 0; return r; }
template <typename V> __device__ __forceinline__ V cmake(double x, double y) {
  V r;
  r.x = (decltype(r.x))x;
  r.y = (decltype(r.y))y;
  return r;
}
template <typename V> __device__ __forceinline__ V cfma(V a, V b, V c) {  // c + a b
  c.x += a.x * b.x - a.y * b.y;
  c.y += a.x * b.y + a.y * b.x;
  return c;
}
template <typename V> __device__ __forceinline__ V cjfma(V a, V b, V c) {  // c + conj(a) b
  c.x += a.x * b.x + a.y * b.y;
  c.y += a.x * b.y - a.y * b.x;
  return c;
}

// 1. c_s[b][u] by linear interpolation of csi[g][b][u] along the pilots of u
template <typename T>
__global__ void interp_kernel(const float2 *csi, typename CT<T>::V *H, uint32_t M, uint32_t K,
                              uint32_t S, uint32_t sg, uint32_t G) {
  using V = typename CT<T>::V;
  const uint64_t total = (uint64_t)S * M * K;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t u = (uint32_t)(e % K), b = (uint32_t)((e / K) % M), s = (uint32_t)(e / ((uint64_t)K * M));
    const double p = ((double)s - (double)(u % sg)) / (double)sg;  // pilot index coordinate
    int g0 = (int)floor(p);
    g0 = max(0, min(g0, (int)G - 2));
    double t = G > 1 ? p - g0 : 0.0;
    t = fmin(fmax(t, 0.0), 1.0);
    const float2 a = csi[((uint64_t)g0 * M + b) * K + u];
    const float2 c = G > 1 ? csi[((uint64_t)(g0 + 1) * M + b) * K + u] : a;
    H[e] = cmake<V>((1.0 - t) * a.x + t * c.x, (1.0 - t) * a.y + t * c.y);
  }
}

// 2. G_s[u][v] = sum_b c_s[b][u] conj(c_s[b][v]) (the reference's Gram C C^H
// of the CSI, beamform.cu:74-122), one CTA per subcarrier, c_s staged in
// shared memory
template <typename T>
__global__ void gram_kernel(const typename CT<T>::V *H, typename CT<T>::V *Gm, uint32_t M, uint32_t K) {
  using V = typename CT<T>::V;
  extern __shared__ __align__(16) unsigned char gsm[];
  V *h = reinterpret_cast<V *>(gsm);
  const uint32_t s = blockIdx.x;
  const V *Hs = H + (uint64_t)s * M * K;
  for (uint32_t e = threadIdx.x; e < M * K; e += blockDim.x) h[e] = Hs[e];
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < K * K; e += blockDim.x) {
    const uint32_t u = e / K, v = e % K;
    V acc = cz<V>();
    for (uint32_t b = 0; b < M; b++) acc = cjfma(h[b * K + v], h[b * K + u], acc);
    Gm[(uint64_t)s * K * K + e] = acc;
  }
}

// 3. X = G^{-1} for matrices src[idx[i]] (or i when idx is null) by
// Gauss-Jordan on [G | I] without pivoting (G is Hermitian positive
// definite), one CTA per matrix, rows in shared memory; flag[i] = 1 when a
// pivot is not positive
template <typename T>
__global__ void inverse_kernel(const typename CT<T>::V *src, const uint32_t *idx,
                               typename CT<T>::V *X, uint32_t K, int *flag) {
  using V = typename CT<T>::V;
  extern __shared__ __align__(16) unsigned char ism[];
  V *A = reinterpret_cast<V *>(ism);  // K x 2K
  __shared__ int bad;
  const uint32_t i = blockIdx.x, m = idx ? idx[i] : i;
  const V *Gm = src + (uint64_t)m * K * K;
  const uint32_t W = 2 * K;
  if (threadIdx.x == 0) bad = 0;
  for (uint32_t e = threadIdx.x; e < K * W; e += blockDim.x) {
    const uint32_t r = e / W, c = e % W;
    A[e] = c < K ? Gm[r * K + c] : cmake<V>(c - K == r ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (uint32_t k = 0; k < K; k++) {
    const T p = A[k * W + k].x;
    if (!(p > (T)0)) {
      if (threadIdx.x == 0) bad = 1;
      break;  // uniform: every thread read the same pivot
    }
    const T inv = (T)1 / p;
    __syncthreads();  // all threads have read the pivot
    for (uint32_t c = threadIdx.x; c < W; c += blockDim.x) {
      V v = A[k * W + c];
      v.x *= inv;
      v.y *= inv;
      A[k * W + c] = v;
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < K * W; e += blockDim.x) {
      const uint32_t r = e / W, c = e % W;
      if (r == k || c == k) continue;  // column k is cleared below
      const V f = A[r * W + k];
      const V rk = A[k * W + c];
      V v = A[r * W + c];
      v.x -= f.x * rk.x - f.y * rk.y;
      v.y -= f.x * rk.y + f.y * rk.x;
      A[r * W + c] = v;
    }
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < K; r += blockDim.x)
      if (r != k) A[r * W + k] = cz<V>();
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0 && flag) flag[i] = bad;
  for (uint32_t e = threadIdx.x; e < K * K; e += blockDim.x)
    X[(uint64_t)i * K * K + e] = A[(e / K) * W + K + e % K];
}

// ||I - G_s X_s||_F per subcarrier
__global__ void residual_kernel(const float2 *Gm, const float2 *X, float *res, uint32_t K, uint32_t S) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  const float2 *g = Gm + (uint64_t)s * K * K, *x = X + (uint64_t)s * K * K;
  float acc = 0.f;
  for (uint32_t r = 0; r < K; r++)
    for (uint32_t c = 0; c < K; c++) {
      float2 v = make_float2(r == c ? -1.f : 0.f, 0.f);
      for (uint32_t k = 0; k < K; k++) v = cfma(g[r * K + k], x[k * K + c], v);
      acc += v.x * v.x + v.y * v.y;
    }
  res[s] = sqrtf(acc);
}

// training targets: A [S][4][4], b [S][4] from the FP64 centre inverses Yc
// and the FP64 per-subcarrier inverses Xs
__global__ void targets_kernel(const double2 *Yc, const double2 *Xs, float *A, float *bv, uint32_t K,
                               uint32_t S, uint32_t sg, uint32_t G) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  const uint32_t g = s / sg, KK = K * K;
  const double2 *Y[kBlend];
  for (int j = 0; j < kBlend; j++) Y[j] = Yc + (uint64_t)min(max((int)g + j - 1, 0), (int)G - 1) * KK;
  const double2 *x = Xs + (uint64_t)s * KK;
  double nx = 0.0;
  for (uint32_t e = 0; e < KK; e++) nx += x[e].x * x[e].x + x[e].y * x[e].y;
  const double inv = nx > 0.0 ? 1.0 / nx : 0.0;
  for (int j = 0; j < kBlend; j++) {
    double bj = 0.0;
    for (uint32_t e = 0; e < KK; e++) bj += Y[j][e].x * x[e].x + Y[j][e].y * x[e].y;
    bv[(uint64_t)s * kBlend + j] = (float)(bj * inv);
    for (int k = j; k < kBlend; k++) {
      double a = 0.0;
      for (uint32_t e = 0; e < KK; e++) a += Y[j][e].x * Y[k][e].x + Y[j][e].y * Y[k][e].y;
      A[((uint64_t)s * kBlend + j) * kBlend + k] = (float)(a * inv);
      A[((uint64_t)s * kBlend + k) * kBlend + j] = (float)(a * inv);
    }
  }
}

// interpolation position of subcarrier s for user u: c_s = (1 - t) csi[g0]
// + t csi[g0 + 1] (integer floor division, then one float division)
__device__ __forceinline__ void interp_pos(uint32_t s, uint32_t u, uint32_t sg, uint32_t G, int &g0,
                                           float &t) {
  const int num = (int)s - (int)(u % sg);
  int q = num >= 0 ? num / (int)sg : -(((-num) + (int)sg - 1) / (int)sg);
  const int gmax = (int)G - 2;
  g0 = max(0, min(q, gmax));
  t = G > 1 ? fminf(fmaxf((float)(num - g0 * (int)sg) / (float)sg, 0.f), 1.f) : 0.f;
}

// Rows of the CSI staged in shared memory are ldc(K) long: the next even
// number (16-byte loads of two users), plus one 16-byte chunk from K = 8 on, so
// that neighbouring antennas sit in different banks; one user stays one.
__host__ __device__ constexpr uint32_t ldc_of(uint32_t K) {
  return K == 1 ? 1 : (K + 1) / 2 * 2 + (K < 8 ? 0 : 2);
}
// The K x K matrices are padded with zeros to KP x KP (KP the power of two from
// 4 on that holds K), rows of ldm(KP): a 16-byte chunk more, for the same reason.
__host__ __device__ constexpr uint32_t ldm_of(uint32_t KP) { return KP + 2; }

// elements i and i + 1 (vec: i is even and a 16-byte load will do)
__device__ __forceinline__ float4 pair_at(const float2 *p, bool vec) {
  if (vec) return *reinterpret_cast<const float4 *>(p);
  return make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
}

// c_s [M][ldc] of subcarrier s into shared memory; ig / iw: per (s, u) the
// lower pilot group and the weight of the upper one (interp_pos, tabulated).
// A thread keeps one user; the element past a row's users is 0 for K odd.
template <int KP>
__device__ __forceinline__ void interp_smem(const float2 *csi, const int *ig, const float *iw, float2 *c,
                                            uint32_t s, uint32_t M, uint32_t K, uint32_t G, uint32_t ldc) {
  constexpr uint32_t step = 256 / KP;
  const uint32_t u = threadIdx.x % KP, b0 = threadIdx.x / KP;
  if (u >= K) {
    if (u == K && ldc > K)
      for (uint32_t b = b0; b < M; b += step) c[b * ldc + u] = make_float2(0.f, 0.f);
    return;
  }
  const int g0 = ig[s * K + u];
  const float t = iw[s * K + u];
  const float2 *lo = csi + ((uint64_t)g0 * M + b0) * K + u, *hi = G > 1 ? lo + (uint64_t)M * K : lo;
  float2 *d = c + b0 * ldc + u;
#pragma unroll 8
  for (uint32_t b = b0; b < M; b += step) {
    const float2 a = *lo, e = *hi;
    *d = make_float2((1.f - t) * a.x + t * e.x, (1.f - t) * a.y + t * e.y);
    lo += step * K;
    hi += step * K;
    d += step * ldc;
  }
}

// The Gram of the staged CSI into gm (KP x KP, the padding zero): 2 x 2 outputs
// a thread, the antennas split over up to four groups of threads whose sums
// meet in gm, b1, b2, b3 (a matrix each).  All 256 threads.
template <int KP>
__device__ __forceinline__ void gram_smem(const float2 *c, float2 *gm, float2 *b1, float2 *b2, float2 *b3, uint32_t M,
                                          uint32_t K, uint32_t ldc) {
  constexpr uint32_t T2 = KP / 2, nt = T2 * T2, parts = 256 / nt < 4 ? 256 / nt : 4, ldm = ldm_of(KP);
  const uint32_t tid = threadIdx.x, part = tid / nt, u = tid % nt / T2 * 2, v = tid % T2 * 2;
  const bool vec = ldc % 2 == 0;
  float2 a[2][2] = {{cz<float2>(), cz<float2>()}, {cz<float2>(), cz<float2>()}};
  if (part < parts && u < K && v < K) {
    const float2 *pu = c + part * ldc + u, *pv = c + part * ldc + v;
#pragma unroll 4
    for (uint32_t b = part; b < M; b += parts) {
      const float4 cu = pair_at(pu, vec), cv = pair_at(pv, vec);
      const float2 u0 = make_float2(cu.x, cu.y), u1 = make_float2(cu.z, cu.w);
      const float2 v0 = make_float2(cv.x, cv.y), v1 = make_float2(cv.z, cv.w);
      a[0][0] = cjfma(v0, u0, a[0][0]);
      a[0][1] = cjfma(v1, u0, a[0][1]);
      a[1][0] = cjfma(v0, u1, a[1][0]);
      a[1][1] = cjfma(v1, u1, a[1][1]);
      pu += parts * ldc;
      pv += parts * ldc;
    }
  }
  if (part < parts) {
    float2 *d = part == 0 ? gm : part == 1 ? b1 : part == 2 ? b2 : b3;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
        d[(u + i) * ldm + v + j] = u + i < K && v + j < K ? a[i][j] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  if (parts > 1) {
    for (uint32_t e = tid; e < KP * KP; e += 256) {
      const uint32_t o = e / KP * ldm + e % KP;
      float2 s = gm[o];
      for (uint32_t q = 1; q < parts; q++) {
        const float2 w = (q == 1 ? b1 : q == 2 ? b2 : b3)[o];
        s.x += w.x;
        s.y += w.y;
      }
      gm[o] = s;
    }
    __syncthreads();
  }
}

// gj_inverse for any KP here (its smallest grid is 16 x 16)
template <int KP>
__device__ __forceinline__ bool inverse_smem(const float2 *G, float2 *X, uint32_t K, float2 *prow, int *bad) {
  constexpr uint32_t ldm = ldm_of(KP);
  return KP <= 16 ? gj_inverse<16>(G, X, K, ldm, prow, bad) : gj_inverse<32>(G, X, K, ldm, prow, bad);
}

__global__ void interp_table_kernel(int *ig, float *iw, uint32_t K, uint32_t S, uint32_t sg, uint32_t G) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= S * K) return;
  int g0;
  float t;
  interp_pos(e / K, e % K, sg, G, g0, t);
  ig[e] = g0;
  iw[e] = t;
}

// The Gram at each group's centre subcarrier and its inverse, a CTA per group
template <int KP>
__global__ void __launch_bounds__(256) centre_kernel(const float2 *csi, const int *ig, const float *iw,
                                                     const uint32_t *cidx, float2 *Gc, float2 *Xc, uint32_t M,
                                                     uint32_t K, uint32_t G, int *flag) {
  extern __shared__ __align__(16) unsigned char sgm[];
  __shared__ int bad;
  pdl_wait();
  constexpr uint32_t ldm = ldm_of(KP), mat = KP * ldm;
  const uint32_t g = blockIdx.x, KK = K * K, ldc = ldc_of(K);
  float2 *gm = reinterpret_cast<float2 *>(sgm), *b1 = gm + mat, *b2 = b1 + mat, *b3 = b2 + mat, *c = b3 + mat;
  float2 *prow = c + M * ldc + 2;
  if (threadIdx.x == 0) bad = 0;
  interp_smem<KP>(csi, ig, iw, c, cidx[g], M, K, G, ldc);
  __syncthreads();
  gram_smem<KP>(c, gm, b1, b2, b3, M, K, ldc);
  const bool ok = inverse_smem<KP>(gm, b1, K, prow, &bad);
  if (threadIdx.x == 0 && flag) flag[g] = ok ? 0 : 1;
  for (uint32_t e = threadIdx.x; e < KK; e += 256) {
    const uint32_t o = e / K * ldm + e % K;
    Gc[(uint64_t)g * KK + e] = gm[o];
    Xc[(uint64_t)g * KK + e] = b1[o];
  }
}

// per group g: ||Gc[g]||_F, and for j = -1, +1, +2 the relative distance
// ||Gc[g+j] - Gc[g]|| / ||Gc[g]|| and trace ratio minus 1 -> st[g][6]
__global__ void group_stats_kernel(const float2 *Gc, float *st, uint32_t K, uint32_t G) {
  __shared__ float red[8][256];
  const uint32_t g = blockIdx.x, KK = K * K;
  const float2 *C0 = Gc + (uint64_t)g * KK;
  const int js[3] = {-1, 1, 2};
  float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // n0, t0, d[-1], d[1], d[2], t[-1], t[1], t[2]
  for (uint32_t e = threadIdx.x; e < KK; e += blockDim.x) {
    const float2 a = C0[e];
    const bool diag = e / K == e % K;
    v[0] += a.x * a.x + a.y * a.y;
    if (diag) v[1] += a.x;
    for (int q = 0; q < 3; q++) {
      const int gj = (int)g + js[q];
      if (gj < 0 || gj >= (int)G) continue;
      const float2 b = Gc[(uint64_t)gj * KK + e];
      v[2 + q] += (b.x - a.x) * (b.x - a.x) + (b.y - a.y) * (b.y - a.y);
      if (diag) v[5 + q] += b.x;
    }
  }
  for (int i = 0; i < 8; i++) red[i][threadIdx.x] = v[i];
  __syncthreads();
  for (uint32_t o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int i = 0; i < 8; i++) red[i][threadIdx.x] += red[i][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float n0 = sqrtf(red[0][0]), t0 = red[1][0];
    for (int q = 0; q < 3; q++) {
      const int gj = (int)g + js[q];
      const bool in = gj >= 0 && gj < (int)G;
      st[g * 6 + q] = in && n0 > 0.f ? sqrtf(red[2 + q][0]) / n0 : 0.f;
      st[g * 6 + 3 + q] = in && t0 > 0.f ? red[5 + q][0] / t0 - 1.f : 0.f;
    }
  }
}

// features [S][sg + 6]: one-hot offset, then the group's six statistics
__global__ void features2_kernel(const float *st, float *F, uint32_t S, uint32_t sg) {
  const uint32_t nf = sg + 6;
  const uint64_t total = (uint64_t)S * nf;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t s = (uint32_t)(e / nf), f = (uint32_t)(e % nf);
    F[e] = f < sg ? (f == s % sg ? 1.f : 0.f) : st[(s / sg) * 6 + (f - sg)];
  }
}

// per subcarrier: interpolated CSI, its Gram (kept for the residual
// diagnostic), the initial iterate (coarse / learned blend / exact
// Gauss-Jordan), Newton-Schulz steps, then the detector W_s = X C, all in
// shared memory with the CSI staged once; X is also stored for the residual.
// Bound by instruction issue (FP32 products of small matrices), so the Gram and
// W take 2 x 2 and 2 x 4 outputs a thread with 16-byte loads and the K x K
// products run over the compile-time padding KP.  1200 subcarriers of 128 x 16,
// two steps: 24 us for a Gram kernel and 43 us for the rest, an output a
// thread; 50 us for both with run-time K, 37 us here.
template <int KP>
__global__ void __launch_bounds__(256, 4) sub_detect_kernel(const float2 *csi, const int *ig, const float *iw,
                                                         float2 *Gm, const float2 *Xc, const float *alpha, int mode,
                                                         uint32_t iters, float2 *Xout, float2 *W, uint32_t M,
                                                         uint32_t K, uint32_t sg, uint32_t G, int *flag) {
  extern __shared__ __align__(16) unsigned char dsm[];
  pdl_wait();
  __shared__ int bad;
  __shared__ float e0sq;  // ||I - G X0||_F^2 of the initial iterate
  constexpr uint32_t ldm = ldm_of(KP), mat = KP * ldm;
  constexpr uint32_t NR = KP == 32 ? 4 : 1, rstep = 256 / KP;  // outputs a thread in a K x K product, rows apart
  const uint32_t KK = K * K, ldc = ldc_of(K), tid = threadIdx.x;
  float2 *g = reinterpret_cast<float2 *>(dsm), *x = g + mat, *t = x + mat, *r4 = t + mat;
  float2 *c = r4 + mat, *prow = c + M * ldc + 2;
  const uint32_t s = blockIdx.x, grp = s / sg;
  const uint32_t q = tid % KP, r0 = tid / KP;  // this thread's outputs (r0 + rstep i, q); r0 >= KP: none
  if (tid == 0) {
    bad = 0;
    e0sq = 0.f;
  }
  interp_smem<KP>(csi, ig, iw, c, s, M, K, G, ldc);
  __syncthreads();
  gram_smem<KP>(c, g, x, t, r4, M, K, ldc);
#pragma unroll
  for (uint32_t i = 0; i < NR; i++) {
    const uint32_t r = r0 + i * rstep;
    if (r < K && q < K) Gm[(uint64_t)s * KK + r * K + q] = g[r * ldm + q];
  }
  if (mode == 2) {
    const bool ok = inverse_smem<KP>(g, x, K, prow, &bad);
    if (tid == 0 && flag) flag[s] = ok ? 0 : 1;
  }
  // the start (or, exact, X's padding)
#pragma unroll
  for (uint32_t i = 0; i < NR; i++) {
    const uint32_t r = r0 + i * rstep, e = r * K + q;
    if (r >= KP) break;
    float2 acc = make_float2(0.f, 0.f);
    if (r < K && q < K) {
      if (mode == 2) continue;
      if (mode == 0) {
        acc = Xc[(uint64_t)grp * KK + e];
      } else {
#pragma unroll
        for (int j = 0; j < kBlend; j++) {
          const int gj = min(max((int)grp + j - 1, 0), (int)G - 1);
          const float a = alpha[(uint64_t)s * kBlend + j];
          const float2 v = Xc[(uint64_t)gj * KK + e];
          acc.x += a * v.x;
          acc.y += a * v.y;
        }
      }
    }
    x[r * ldm + q] = acc;
  }
  if (mode != 2 && tid == 0 && flag) flag[s] = 0;
  __syncthreads();
  // row r of A times column q of B, over the padding too
  auto product = [&](const float2 *A, const float2 *B, float2 (&acc)[NR]) {
#pragma unroll
    for (uint32_t i = 0; i < NR; i++) acc[i] = make_float2(0.f, 0.f);
    if (r0 >= KP) return;
#pragma unroll
    for (uint32_t k = 0; k < KP; k += 2) {
      const float2 b0 = B[k * ldm + q], b1 = B[(k + 1) * ldm + q];
#pragma unroll
      for (uint32_t i = 0; i < NR; i++) {
        const float4 a = *reinterpret_cast<const float4 *>(A + (r0 + i * rstep) * ldm + k);
        acc[i] = cfma(make_float2(a.x, a.y), b0, acc[i]);
        acc[i] = cfma(make_float2(a.z, a.w), b1, acc[i]);
      }
    }
  };
  for (uint32_t it = 0; it < iters; it++) {
    float2 acc[NR];
    float part = 0.f;
    product(g, x, acc);
#pragma unroll
    for (uint32_t i = 0; i < NR; i++) {
      const uint32_t r = r0 + i * rstep;
      if (r >= KP) break;
      t[r * ldm + q] = make_float2((r == q ? 2.f : 0.f) - acc[i].x, -acc[i].y);
      const float ex = (r == q ? 1.f : 0.f) - acc[i].x;
      if (r < K && q < K) part += ex * ex + acc[i].y * acc[i].y;
    }
    if (it == 0 && mode != 2) {
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if ((tid & 31) == 0) atomicAdd(&e0sq, part);
    }
    __syncthreads();
    if (it == 0 && mode != 2 && !(e0sq < 1.f)) {
      // Newton-Schulz converges only from ||I - G X0|| < 1: a start further
      // off (the blend of neighbouring groups' inverses under a channel that
      // changes too fast across the band) takes the exact inverse instead,
      // flagged 2 (uniform: every thread read the same sum)
      const bool ok = inverse_smem<KP>(g, x, K, prow, &bad);
      if (tid == 0 && flag) flag[s] = ok ? 2 : 1;
      break;
    }
    product(x, t, acc);
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < NR; i++)
      if (r0 + i * rstep < KP) x[(r0 + i * rstep) * ldm + q] = acc[i];
    __syncthreads();
  }
  // X transposed into t (t[v][u]): a thread's two users are neighbours
#pragma unroll
  for (uint32_t i = 0; i < NR; i++) {
    const uint32_t r = r0 + i * rstep;
    if (r >= KP) break;
    const float2 v = x[r * ldm + q];
    if (r < K && q < K) Xout[(uint64_t)s * KK + r * K + q] = v;
    t[q * ldm + r] = v;
  }
  __syncthreads();
  constexpr uint32_t T2 = KP / 2, nq = 256 / T2;
  const uint32_t u = tid % T2 * 2, bq = tid / T2;
  const bool vc = ldc % 2 == 0, two = u + 1 < K, w16 = K % 2 == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0;
  if (u >= K) return;
  for (uint32_t b0 = bq; b0 < M; b0 += 4 * nq) {
    float2 a[4][2];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i][0] = a[i][1] = make_float2(0.f, 0.f);
    const float2 *xr = t + u, *cr[4];
#pragma unroll
    for (int i = 0; i < 4; i++) cr[i] = c + min(b0 + i * nq, M - 1) * ldc;
    auto step = [&](const float4 &xv, const float2 (&cv)[4]) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        a[i][0] = cfma(make_float2(xv.x, xv.y), cv[i], a[i][0]);
        a[i][1] = cfma(make_float2(xv.z, xv.w), cv[i], a[i][1]);
      }
    };
    uint32_t v = 0;
    if (vc)
#pragma unroll 4
      for (; v + 1 < K; v += 2) {
        float2 c0[4], c1[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float4 w = *reinterpret_cast<const float4 *>(cr[i] + v);
          c0[i] = make_float2(w.x, w.y);
          c1[i] = make_float2(w.z, w.w);
        }
        step(*reinterpret_cast<const float4 *>(xr + v * ldm), c0);
        step(*reinterpret_cast<const float4 *>(xr + (v + 1) * ldm), c1);
      }
    for (; v < K; v++) {
      float2 c0[4];
#pragma unroll
      for (int i = 0; i < 4; i++) c0[i] = cr[i][v];
      step(*reinterpret_cast<const float4 *>(xr + v * ldm), c0);
    }
    float2 *w = W + ((uint64_t)s * M + b0) * K + u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (b0 + i * nq >= M) break;
      if (w16) {
        *reinterpret_cast<float4 *>(w) = make_float4(a[i][0].x, a[i][0].y, a[i][1].x, a[i][1].y);
      } else {
        w[0] = a[i][0];
        if (two) w[1] = a[i][1];
      }
      w += nq * K;
    }
  }
}

unsigned grid_for(uint64_t n) { return (unsigned)std::min<uint64_t>((n + 255) / 256, 148ull * 16); }

}  // namespace
}  // namespace mb

using namespace mb;


struct mb_lzf {
  uint32_t M, K, S, sg, G;
  float2 *Gs, *Gc, *Xc, *X;       // FP32 working set: per-subcarrier and centre Grams, inverses
  float *feat, *alpha, *res, *stats;  // stats: per-group feature statistics [G][6]
  uint32_t *cidx;                 // centre subcarrier of each group
  int *ig;                        // [S][K] lower pilot group of the interpolation
  float *iw;                      // [S][K] weight of the upper pilot group
  int *flag;                      // per-inverse non-PD flags
  double2 *H64, *Gs64, *Yc64, *X64;  // FP64 training-target set (allocated on first use)
};

extern "C" mb_status mb_lzf_destroy(mb_lzf *z) {
  if (!z) return MB_BAD_ARG;
  for (void *p : {(void *)z->ig, (void *)z->iw, (void *)z->stats, (void *)z->Gs, (void *)z->Gc, (void *)z->Xc, (void *)z->X,
                  (void *)z->feat, (void *)z->alpha, (void *)z->res, (void *)z->cidx, (void *)z->flag,
                  (void *)z->H64, (void *)z->Gs64, (void *)z->Yc64, (void *)z->X64})
    cudaFree(p);
  delete z;
  return MB_OK;
}

extern "C" mb_status mb_lzf_create(uint32_t M, uint32_t K, uint32_t S, uint32_t sg, mb_lzf **out) {
  if (!out) return MB_BAD_ARG;
  *out = nullptr;
  if (M == 0 || K == 0 || K > 32 || K > M || S == 0 || sg == 0 || sg > 64) return MB_BAD_SHAPE;
  mb_lzf *z = new mb_lzf();
  z->M = M;
  z->K = K;
  z->S = S;
  z->sg = sg;
  z->G = (S + sg - 1) / sg;
  mb_status st = MB_OK;
  auto alloc = [&](void **p, size_t bytes) {
    if (st != MB_OK) return;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) st = record_error(e);
  };
  const size_t skk = (size_t)S * K * K, gkk = (size_t)z->G * K * K;
  alloc((void **)&z->Gs, sizeof(float2) * skk);
  alloc((void **)&z->X, sizeof(float2) * skk);
  alloc((void **)&z->Gc, sizeof(float2) * gkk);
  alloc((void **)&z->Xc, sizeof(float2) * gkk);
  alloc((void **)&z->feat, sizeof(float) * (size_t)S * (sg + 6));
  alloc((void **)&z->alpha, sizeof(float) * (size_t)S * kBlend);
  alloc((void **)&z->res, sizeof(float) * S);
  alloc((void **)&z->stats, sizeof(float) * 6 * z->G);
  alloc((void **)&z->ig, sizeof(int) * (size_t)S * K);
  alloc((void **)&z->iw, sizeof(float) * (size_t)S * K);
  if (st == MB_OK) {
    interp_table_kernel<<<(S * K + 255) / 256, 256>>>(z->ig, z->iw, K, S, sg, z->G);
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) st = record_error(e);
  }
  alloc((void **)&z->cidx, sizeof(uint32_t) * z->G);
  alloc((void **)&z->flag, sizeof(int) * std::max(z->G, S));
  if (st == MB_OK) {
    std::vector<uint32_t> c(z->G);
    for (uint32_t g = 0; g < z->G; g++) c[g] = std::min(g * sg + sg / 2, S - 1);
    cudaError_t e = cudaMemcpy(z->cidx, c.data(), sizeof(uint32_t) * z->G, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) st = record_error(e);
  }
  if (st != MB_OK) {
    mb_lzf_destroy(z);
    return st;
  }
  *out = z;
  return MB_OK;
}

extern "C" uint32_t mb_lzf_num_features(uint32_t sg) { return sg + 6; }

static uint32_t kp_of(uint32_t K) { return K <= 4 ? 4 : K <= 8 ? 8 : K <= 16 ? 16 : 32; }
// the kernel template for K users
#define MB_LZF_OF(kernel, K) \
  (kp_of(K) == 4 ? kernel<4> : kp_of(K) == 8 ? kernel<8> : kp_of(K) == 16 ? kernel<16> : kernel<32>)

// four matrices, the staged CSI and the pivot rows of the inverse
static size_t detect_smem(const mb_lzf *z) {
  const uint32_t KP = kp_of(z->K);
  return sizeof(float2) * (4 * (size_t)KP * ldm_of(KP) + (size_t)z->M * ldc_of(z->K) + 2 + 64);
}

// centre Grams and their inverses (FP32)
static mb_status lzf_front(mb_lzf *z, const mb_c32 *csi, cudaStream_t st) {
  const uint32_t M = z->M, K = z->K;
  MB_CUDA_TRY(pdl_launch(MB_LZF_OF(centre_kernel, K), z->G, 256, detect_smem(z), st,
                         reinterpret_cast<const float2 *>(csi), z->ig, z->iw, z->cidx, z->Gc, z->Xc, M, K, z->G, z->flag));
  return MB_OK;
}

// The kernels that stage one subcarrier's M x K CSI in shared memory take
// up to the device's opt-in limit (raised once per device): 256 x 32 needs
// 101 KB (detector) and 128 KB (FP64 Gram of the targets).
static mb_status lzf_configure(size_t *limit) {
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> lim[64] = {};
  int dev = 0, maxs = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (!(configured.load() & bit)) {
    MB_CUDA_TRY(cudaDeviceGetAttribute(&maxs, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    int l = maxs;
    const void *ks[] = {(const void *)centre_kernel<4>,      (const void *)centre_kernel<8>,
                        (const void *)centre_kernel<16>,     (const void *)centre_kernel<32>,
                        (const void *)sub_detect_kernel<4>,  (const void *)sub_detect_kernel<8>,
                        (const void *)sub_detect_kernel<16>, (const void *)sub_detect_kernel<32>,
                        (const void *)gram_kernel<double>};
    for (const void *k : ks) {
      cudaFuncAttributes fa;
      MB_CUDA_TRY(cudaFuncGetAttributes(&fa, k));
      MB_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, maxs - (int)fa.sharedSizeBytes));
      l = std::min(l, maxs - (int)fa.sharedSizeBytes);
    }
    lim[dev & 63].store(l);
    configured.fetch_or(bit);
  }
  *limit = (size_t)lim[dev & 63].load();
  return MB_OK;
}

static mb_status lzf_shared_mem_ok(const mb_lzf *z) {
  // one subcarrier's M x K CSI is staged in shared memory (FP64 for targets)
  size_t limit = 0;
  const mb_status r = lzf_configure(&limit);
  if (r != MB_OK) return r;
  return (size_t)z->M * z->K * sizeof(double2) <= limit && detect_smem(z) <= limit ? MB_OK : MB_UNSUPPORTED;
}

// the network's inputs from the centre Grams, as rows in memory
static mb_status lzf_features_of(mb_lzf *z, float *features, cudaStream_t st) {
  group_stats_kernel<<<z->G, 256, 0, st>>>(z->Gc, z->stats, z->K, z->G);
  features2_kernel<<<grid_for((uint64_t)z->S * (z->sg + 6)), 256, 0, st>>>(z->stats, features, z->S, z->sg);
  MB_CUDA_TRY(cudaGetLastError());
  return MB_OK;
}

extern "C" mb_status mb_lzf_features(mb_lzf *z, const mb_c32 *csi, float *features, void *stream) {
  if (!z || !csi || !features) return MB_BAD_ARG;
  if (lzf_shared_mem_ok(z) != MB_OK) return MB_UNSUPPORTED;
  cudaStream_t st = as_stream(stream);
  mb_status r = lzf_front(z, csi, st);
  if (r != MB_OK) return r;
  return lzf_features_of(z, features, st);
}

extern "C" mb_status mb_lzf_run(mb_lzf *z, const mb_c32 *csi, mb_mlp *mlp, int init,
                                uint32_t ns_iters, mb_c32 *W, void *stream) {
  if (!z || !csi || !W) return MB_BAD_ARG;
  if (init < MB_LZF_COARSE || init > MB_LZF_EXACT || (init == MB_LZF_LEARNED && !mlp)) return MB_BAD_ARG;
  if (lzf_shared_mem_ok(z) != MB_OK) return MB_UNSUPPORTED;
  cudaStream_t st = as_stream(stream);
  const uint32_t M = z->M, K = z->K, S = z->S;
  mb_status r = lzf_front(z, csi, st);
  if (r != MB_OK) return r;
  if (init == MB_LZF_LEARNED) {
    // the network's kernel forms its inputs itself where its shape allows
    r = mlp_forward_features(mlp, BlendFeatures{z->Gc, z->sg, K, z->G}, S, z->alpha, st);
    if (r == MB_UNSUPPORTED) {
      r = lzf_features_of(z, z->feat, st);
      if (r == MB_OK) r = mb_mlp_forward(mlp, z->feat, S, z->alpha, st);
    }
    if (r != MB_OK) return r;
  }
  const size_t smem = detect_smem(z);
  MB_CUDA_TRY(pdl_launch(MB_LZF_OF(sub_detect_kernel, K), S, 256, smem, st, reinterpret_cast<const float2 *>(csi), z->ig,
                         z->iw, z->Gs, z->Xc, init == MB_LZF_LEARNED ? z->alpha : nullptr, init, ns_iters, z->X,
                         reinterpret_cast<float2 *>(W), M, K, z->sg, z->G, z->flag));
  return MB_OK;
}

extern "C" mb_status mb_lzf_flags(mb_lzf *z, int32_t *flags, void *stream) {
  if (!z || !flags) return MB_BAD_ARG;
  MB_CUDA_TRY(cudaMemcpyAsync(flags, z->flag, sizeof(int) * z->S, cudaMemcpyDeviceToDevice, as_stream(stream)));
  return MB_OK;
}

extern "C" mb_status mb_lzf_residual(mb_lzf *z, float *res, void *stream) {
  if (!z || !res) return MB_BAD_ARG;
  residual_kernel<<<(z->S + 127) / 128, 128, 0, as_stream(stream)>>>(z->Gs, z->X, res, z->K, z->S);
  MB_CUDA_TRY(cudaGetLastError());
  return MB_OK;
}

extern "C" mb_status mb_lzf_targets(mb_lzf *z, const mb_c32 *csi, float *A, float *b, void *stream) {
  if (!z || !csi || !A || !b) return MB_BAD_ARG;
  if (lzf_shared_mem_ok(z) != MB_OK) return MB_UNSUPPORTED;
  cudaStream_t st = as_stream(stream);
  const uint32_t M = z->M, K = z->K, S = z->S;
  if (!z->H64) {
    const size_t smk = (size_t)S * M * K, skk = (size_t)S * K * K, gkk = (size_t)z->G * K * K;
    MB_CUDA_TRY(cudaMalloc(&z->H64, sizeof(double2) * smk));
    MB_CUDA_TRY(cudaMalloc(&z->Gs64, sizeof(double2) * skk));
    MB_CUDA_TRY(cudaMalloc(&z->X64, sizeof(double2) * skk));
    MB_CUDA_TRY(cudaMalloc(&z->Yc64, sizeof(double2) * gkk));
  }
  interp_kernel<double><<<grid_for((uint64_t)S * M * K), 256, 0, st>>>(
      reinterpret_cast<const float2 *>(csi), z->H64, M, K, S, z->sg, z->G);
  gram_kernel<double><<<S, 256, sizeof(double2) * M * K, st>>>(z->H64, z->Gs64, M, K);
  inverse_kernel<double><<<S, 256, sizeof(double2) * 2 * K * K, st>>>(z->Gs64, nullptr, z->X64, K, z->flag);
  inverse_kernel<double><<<z->G, 256, sizeof(double2) * 2 * K * K, st>>>(z->Gs64, z->cidx, z->Yc64, K,
                                                                        nullptr);
  targets_kernel<<<(S + 127) / 128, 128, 0, st>>>(z->Yc64, z->X64, A, b, K, S, z->sg, z->G);
  MB_CUDA_TRY(cudaGetLastError());
  return MB_OK;
}
