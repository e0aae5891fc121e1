// zf_fp64.cuh -- the FP64 solve of one group, the fallback of both
// mixed-precision detector kernels (zf_mixed.cu, zf_direct.cu), and the
// detector image's layout.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"
#include "zf_ldl.cuh"

namespace mb {

constexpr uint32_t kZfTile = 64;  // antennas per k tile of the image

__device__ __forceinline__ uint32_t img_off(uint32_t r, uint32_t kk, uint32_t MM) {
  // canonical K-major, no swizzle: [k tile][row group][k chunk][row][8]
  const uint32_t kt = kk / kZfTile, kin = kk % kZfTile;
  return kt * (MM * kZfTile * 2) + (r / 8) * 1024 + (kin / 8) * 128 + (r % 8) * 16 + (kin % 8) * 2;
}

// antennas of a group in shared memory at a time, at least: odd (any T is), so
// that neighbouring users of one antenna sit in different banks, and small enough
// for the regions that a kernel has to spare (496 K bytes)
constexpr uint32_t kFp64Tile = 31;
__host__ __device__ constexpr uint32_t zf_fp64_tile_bytes(uint32_t K) { return kFp64Tile * K * 16; }

struct Fp64Group {
  int status;  // 2, or 1 (not positive definite, W zero)
  float wmax;  // max |W| of the values this thread stored
};

// Group of cg [M][K] in FP64 (Gram, L D L^H, two products) by the 256 threads:
// W (FP32) over cg and the detector image imgw (MM rows, nkt k tiles).  In shared
// memory Gd [K][K+1], Ct [K][T] (at least 2 KP) and *flag; K <= KP, T odd.
// The columns of C pass through Ct, T antennas at a time, and all 256 threads
// share them.  A thread per antenna with its column in local memory walked K^2
// dependent steps, from L2 where two CTAs left an SM little L1 (and shared memory
// cut to one CTA, 294 us, kept other launches off the SM: six cells of 33 to 64
// users 234 -> 295 us).  75 groups, all in FP64, before / now: 64 x 64 425 / 189
// us, 128 x 64 480 / 226, 128 x 32 133 / 80, 256 x 16 66 / 53.
template <int KP>
__device__ __forceinline__ Fp64Group zf_fp64_group(float2 *cg, uint8_t *imgw, double2 *Gd, double2 *Ct, uint32_t T,
                                                   int *flag, uint32_t M, uint32_t K, uint32_t Mp, uint32_t MM,
                                                   uint32_t nkt) {
  using C = Cplx<double>;
  constexpr uint32_t nt = 256;
  constexpr int GT = KP / 16;
  const uint32_t tid = threadIdx.x, lda = K + 1;
  float wmx = 0.f;
  const uint32_t db = nt / K, du = nt % K;  // element tid of a tile in (antenna, user) order, then 256 further
  C *A = reinterpret_cast<C *>(Gd), *Cs = reinterpret_cast<C *>(Ct);
  auto each = [&](uint32_t n, auto f) {
    uint32_t b = tid / K, u = tid % K;
    for (uint32_t e = tid; e < n * K; e += nt) {
      f(e, b, u);
      b += db;
      u += du;
      if (u >= K) {
        u -= K;
        b++;
      }
    }
  };
  auto load = [&](uint32_t b0, uint32_t n) {
    const float2 *c = cg + (uint64_t)b0 * K;
    each(n, [&](uint32_t e, uint32_t b, uint32_t u) { Cs[u * T + b] = mk<double>(c[e].x, c[e].y); });
    __syncthreads();
  };
  __syncthreads();  // the caller's reads of *flag and of the two regions
  if (tid == 0) *flag = 0;
  // Gram: the thread's entries (ti + 16 a, tj + 16 b) of the lower blocks, a
  // tile's share added in shared memory (registers for all of them would spill)
  const uint32_t ti = tid / 16, tj = tid % 16;
  for (uint32_t b0 = 0; b0 < M; b0 += T) {
    const uint32_t n = min(T, M - b0);
    load(b0, n);
#pragma unroll
    for (int a = 0; a < GT; a++) {
      const uint32_t i = ti + 16 * a;
      C acc[GT];
      const C *ca = Cs + min(i, K - 1) * T, *cb[GT];
#pragma unroll
      for (int b = 0; b <= a; b++) {
        acc[b] = mk<double>(0.0, 0.0);
        cb[b] = Cs + min(tj + 16 * b, K - 1) * T;
      }
#pragma unroll(GT == 1 ? 4 : 1)
      for (uint32_t m = 0; m < n; m++) {
        const C av = ca[m];
#pragma unroll
        for (int b = 0; b <= a; b++) {
          const C bv = cb[b][m];
          acc[b].x += av.x * bv.x + av.y * bv.y;
          acc[b].y += av.y * bv.x - av.x * bv.y;
        }
      }
#pragma unroll
      for (int b = 0; b <= a; b++) {
        const uint32_t j = tj + 16 * b;
        if (i >= K || j > i) continue;
        C v = acc[b];
        if (b0) v = mk<double>(A[i * lda + j].x + v.x, A[i * lda + j].y + v.y);
        A[i * lda + j] = v;
        if (j < i) A[j * lda + i] = mk<double>(v.x, -v.y);
      }
    }
    __syncthreads();
  }
  ldl_eliminate<double, KP>(A, lda, K, flag, Cs);
  const bool pd = *flag == 0;
  for (uint32_t c = tid; c < nkt * MM * kZfTile * 2 / 16; c += nt)
    reinterpret_cast<uint4 *>(imgw)[c] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (uint32_t b0 = 0; b0 < M; b0 += T) {
    const uint32_t n = min(T, M - b0);
    if (pd) {
      load(b0, n);
      ldl_products<double, KP <= 32 ? 1 : 4>(A, Cs, n, K, T, lda);  // (unrolled, the callers of the call spill)
    }
    each(n, [&](uint32_t e, uint32_t tb, uint32_t u) {
      const uint32_t b = b0 + tb;
      const C v = Cs[u * T + tb];
      const float2 w = pd ? make_float2((float)v.x, (float)v.y) : make_float2(0.f, 0.f);
      cg[(uint64_t)b0 * K + e] = w;
      wmx = fmaxf(wmx, sqrtf(w.x * w.x + w.y * w.y));
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u, b, MM)) = __float2bfloat16_rn(w.x);
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u, Mp + b, MM)) = __float2bfloat16_rn(-w.y);
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u + 1, b, MM)) = __float2bfloat16_rn(w.y);
      *reinterpret_cast<__nv_bfloat16 *>(imgw + img_off(2 * u + 1, Mp + b, MM)) = __float2bfloat16_rn(w.x);
    });
    __syncthreads();
  }
  return {pd ? 2 : 1, wmx};
}

// The same as a call, which leaves the caller's registers alone: in line
// zf_direct.cu's kernel spills 340 bytes a thread instead of 72 and zf_mixed.cu's
// for up to 32 users 44 instead of none. With more users that kernel has it in
// line (205 groups of 256 x 64: 166.7 us a pass of pilots, detector and precoder, 168.7
// as a call).
template <int KP, uint32_t MM>
__device__ __noinline__ Fp64Group zf_fp64_group_call(float2 *cg, uint8_t *imgw, double2 *Gd, double2 *Ct, uint32_t T,
                                                     int *flag, uint32_t M, uint32_t K) {
  const uint32_t Mp = (M + kZfTile - 1) / kZfTile * kZfTile;  // as tc_shape()
  return zf_fp64_group<KP>(cg, imgw, Gd, Ct, T, flag, M, K, Mp, MM, 2 * Mp / kZfTile);
}

}  // namespace mb
