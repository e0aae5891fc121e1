// ldpc.cuh -- the LDPC handle (ldpc.cu), for the slot's decode stage.
#pragma once
#include "common.cuh"

struct mb_ldpc {
  uint32_t kb, Z, mb, nnz, max_batch;
  int dev;
  uint32_t *row_ptr;   // [mb + 1] device
  uint16_t *col, *sh;  // [nnz] device, rows < mb, by (row, col)
  uint32_t *inv;       // device: B^-1's circulants, block row i's entries (block column << 16 | shift)
                       // at inv[i] .. inv[i + 1] - 1
  uint4 *state;        // [(max_batch + 1) / 2][mb][Z] device, per pair of blocks: message magnitudes, signs, who takes the second
};
