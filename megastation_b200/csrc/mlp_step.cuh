// mlp_step.cuh -- the fused training step of the 3-layer MLP (mlp_step.cu).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace mb {

// Shapes that train in one kernel per batch; the weights of a wider network
// do not fit beside its activations in one SM's shared memory.
constexpr uint32_t kStepMaxIn = 64, kStepMaxWidth = 256, kStepMaxOut = 16;
constexpr uint32_t kStepTile = 64;   // samples per CTA pass
constexpr uint32_t kStepSlots = 148; // partial-sum slots (CTAs) at most

struct MlpStepShape {
  uint32_t I, W, O;      // n_in, width, n_out
  uint32_t Ip, Wp;       // n_in to a multiple of 16, width to 128 or 256
  uint64_t off[6];       // flat parameter offsets: W1, b1, W2, b2, W3, b3
  uint64_t n_params;
  uint64_t slot;         // floats per partial-sum slot: n_params gradients and the loss
  // BF16 weight images in shared-memory form: 8 x 8 blocks of 128 bytes, a
  // block row's blocks one after the other, W1 [Ip][Wp], W2 [Wp][Wp], W3 [Wp][16]
  __host__ __device__ uint32_t img2() const { return Ip * Wp; }  // in elements
  __host__ __device__ uint32_t img3() const { return Ip * Wp + Wp * Wp; }
  __host__ __device__ uint32_t img_elems() const { return Ip * Wp + Wp * Wp + Wp * 16; }
};

bool mlp_step_shape(uint32_t I, uint32_t W, uint32_t O, const uint64_t off[6], uint64_t n_params, MlpStepShape *s);
// image element of flat parameter i, or -1 for a bias
__device__ __forceinline__ int mlp_step_img(const MlpStepShape &s, uint64_t i) {
  uint32_t r, c, base, blocks;
  if (i < s.off[1]) {
    r = (uint32_t)i / s.W, c = (uint32_t)i % s.W, base = 0, blocks = s.Wp / 8;
  } else if (i >= s.off[2] && i < s.off[3]) {
    const uint32_t k = (uint32_t)(i - s.off[2]);
    r = k / s.W, c = k % s.W, base = s.img2(), blocks = s.Wp / 8;
  } else if (i >= s.off[4] && i < s.off[5]) {
    const uint32_t k = (uint32_t)(i - s.off[4]);
    r = k / s.O, c = k % s.O, base = s.img3(), blocks = 2;
  } else {
    return -1;
  }
  return (int)(base + (r / 8 * blocks + c / 8) * 64 + r % 8 * 8 + c % 8);
}

// The per-subcarrier blend's features of sample s from the groups' centre Grams
// gc [G][K][K]: one-hot s % sg, then for the neighbours j = -1, 1, 2 of group
// g = s / sg the relative distance ||C_{g+j} - C_g|| / ||C_g|| and the trace
// ratio minus 1 (0 past the band's edges).
struct BlendFeatures {
  const float2 *gc;
  uint32_t sg, K, G;
};
// y [B][O] = the network's outputs for x [B][I], or (x null) for the features
// f (I = f.sg + 6)
cudaError_t mlp_fwd_tc(const MlpStepShape &s, const __nv_bfloat16 *img, const float *params, const float *x,
                       const BlendFeatures &f, uint32_t B, float *y, int *err, cudaStream_t st);
// the same through a network's handle; MB_UNSUPPORTED when its shape does not allow it
mb_status mlp_forward_features(mb_mlp *n, const BlendFeatures &f, uint32_t B, float *y, cudaStream_t st);

// gradients of the batch-mean quadratic loss into g (flat) and, if not null,
// the loss; part: kStepSlots or ceil(B / kStepTile) slots, whichever is fewer
cudaError_t mlp_step(const MlpStepShape &s, const __nv_bfloat16 *img, const float *params, const float *x,
                     const float *A, const float *b, const float *c, uint32_t B, float *part, float *g, float *loss,
                     int *err, cudaStream_t st);

}  // namespace mb
