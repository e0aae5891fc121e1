// noalloc.cu -- the tensor-core equalize entry point for callers that must
// not allocate device memory.
//
// Some hosts cannot call cudaMalloc at the point where they equalize: a
// real-time fronthaul thread that may not block on the driver's allocator,
// a process whose device memory is carved up and fixed at start-up, or an
// embedding framework that owns every allocation itself.  mb_equalize_tc
// asks such callers for two scratch buffers; this variant takes none, and its
// error word is fixed in the library, so a call needs nothing but its inputs
// and outputs.
#include <mutex>

#include "common.cuh"
#include "eq_tc.cuh"

namespace {

// The entry point's limit: the BF16 operands of one symbol (detector images
// of all groups and one symbol's rows) fit in 32 MiB.  No buffer of that size
// stands behind it any more; it stays because hosts choose between this entry
// point and mb_equalize_tc by its MB_TOO_LARGE.
constexpr uint64_t kNoAllocScratchBytes = 32ull << 20;
// The error word of this entry point's kernels (bit 1: a bounded mbarrier
// wait gave up), fixed because the library's own error word is allocated on
// first use.  mb_device_error reports and clears it
// together with that word.
static __device__ int g_noalloc_err;

// Device address of g_noalloc_err per device, looked up once per device with
// that device current.  In host code the word's name is only a handle for the
// runtime, not a device address.  The cached address belongs to the device's
// current context: after cudaDeviceReset it is stale, and this entry point
// must not be called again in that process (as with every other per-device
// table of the library).
std::mutex g_noalloc_mu;
int *g_noalloc_err_addr[64];

}  // namespace

using namespace mb;

// Reads (and optionally clears) this entry point's error word on the current
// device; 0 when the entry point has not run there.
mb_status mb::noalloc_error_word(int *bits, bool clear) {
  *bits = 0;
  int dev = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return MB_OK;
  int *addr = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    addr = g_noalloc_err_addr[dev];
  }
  if (!addr) return MB_OK;
  MB_CUDA_TRY(cudaMemcpy(bits, addr, sizeof(int), cudaMemcpyDeviceToHost));
  if (clear) MB_CUDA_TRY(cudaMemset(addr, 0, sizeof(int)));
  return MB_OK;
}

extern "C" mb_status mb_equalize_tc_noalloc(const mb_c32 *W, const mb_c32 *y, uint32_t K,
                                            uint32_t M, uint32_t S, uint32_t sg,
                                            uint32_t n_sym, uint32_t Qm, uint64_t cb_size,
                                            uint64_t cb_stride, uint64_t zeros,
                                            uint32_t cb_blocks, uint16_t *llr, uint8_t *hard,
                                            const mb_scrambler *scr, mb_c32 *x, void *stream) {
  EqParams p;
  mb_status s = equalize_prepare(p, W, y, K, M, S, sg, n_sym, Qm, cb_size, cb_stride, zeros,
                                 cb_blocks, llr, hard, scr);
  if (s != MB_OK) return s;
  p.x = reinterpret_cast<float2 *>(x);
  if (n_sym == 0) return MB_OK;
  if (!equalize_tc_supported(K, sg, 1)) return MB_UNSUPPORTED;

  const uint64_t G = (S + sg - 1) / sg;
  const uint64_t img_bytes = (G * tc_shape(M, K).img_group_bytes + 255) / 256 * 256;
  const uint64_t sym_bytes = (uint64_t)2 * M * ((S + 7) / 8 * 8) * 2;
  if (img_bytes + sym_bytes > kNoAllocScratchBytes) return MB_TOO_LARGE;

  int dev = 0;
  MB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return MB_UNSUPPORTED;
  int *err = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_err_addr[dev]) {
      void *eaddr = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&eaddr, g_noalloc_err);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return record_error(e);
      }
      g_noalloc_err_addr[dev] = reinterpret_cast<int *>(eaddr);
    }
    err = g_noalloc_err_addr[dev];
  }
  return equalize_tc_c32(p, err, as_stream(stream));
}
