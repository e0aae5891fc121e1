// common.cuh -- shared device/host helpers of the sm_100a baseband library.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/megastation_b200.h"

namespace mb {

// On failure the runtime's sticky "last error" is cleared as well, so that a
// failed API call is reported once and not again by a later launch check.
#define MB_CUDA_TRY(expr)                                   \
  do {                                                      \
    cudaError_t _e = (expr);                                \
    if (_e != cudaSuccess) {                                \
      (void)cudaGetLastError();                             \
      return ::mb::record_error(_e);                        \
    }                                                       \
  } while (0)

#define MB_LAUNCH_CHECK() MB_CUDA_TRY(cudaGetLastError())

mb_status record_error(cudaError_t e);

__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}
__host__ __device__ __forceinline__ float2 cconj(float2 a) {
  return make_float2(a.x, -a.y);
}
// acc += a * b
__device__ __forceinline__ void cfma(float2 &acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.x = fmaf(-a.y, b.y, acc.x);
  acc.y = fmaf(a.x, b.y, acc.y);
  acc.y = fmaf(a.y, b.x, acc.y);
}

// Programmatic dependent launch.  A kernel launched with pdl_launch() is set up
// while the kernel before it in its stream drains and waits in pdl_wait() until
// that one has completed and its writes are visible.  So pdl_wait() is the
// first statement of every thread, before any access to global memory and
// before any return: a CTA that left without it would let the next kernel of
// the chain start with the last but one still running.  Whatever an earlier
// kernel may have written (a caller's buffers too: the writer is the caller's
// last kernel) is read with ordinary loads behind it: __ldg says that the data
// does not change while the kernel is resident, which holds only for tables
// written when their handle was created (twiddles, pilot signs, descrambling
// bytes, the code's B^-1).  It saves 1 to 3 us a
// launch in a chain (pilots to detector of 64 x 16 in FP32, two launches: 16.4
// -> 13.5 us; modulate, precode and inverse FFT of 128 x 16: 26.0 -> 20.4; a
// training step of three: 56 -> 50).  No kernel lets the next one start
// earlier (griddepcontrol.launch_dependents): CTAs placed on whatever SM drains
// first are spread unevenly, which cost more than the overlap gave (FP32
// equalizer of 64 x 16: 10.7 us against 13.9 with it, 32 batched cells 523
// against 626).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// launch of a kernel that calls pdl_wait(); what precedes it in the stream may
// be anything
template <typename... P, typename... A>
inline cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

inline bool is_pow2(uint64_t x) { return x && !(x & (x - 1)); }

inline int ilog2(uint64_t x) {
  int l = 0;
  while ((1ull << l) < x) l++;
  return l;
}

// Per-device table registry (twiddles, scrambler bits).
struct DeviceTables {
  // Stockham twiddle tables per N = 2^l, l in [4, 13]: for each pass p >= 1
  // (radix R, Ns = product of earlier radices) the R x Ns block
  // exp(-2 pi i r k / (Ns R)) at [r][k], blocks concatenated by pass
  float2 *twiddle[14];
  uint32_t *lfsr127_bits;  // 127 bits packed LSB-first in 4 words
  int *err;                // device error word (mb_tc error bits)
};
// for the current device, built once per device under a lock (the QAM maps
// of the modulator are uploaded then too); nullptr on error
const DeviceTables *device_tables();
mb_status upload_mod_tables();  // modscr.cu: QAM maps to the current device

}  // namespace mb
