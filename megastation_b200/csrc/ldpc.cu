// ldpc.cu -- NR LDPC encode and layered min-sum decode over a caller-supplied
// base graph (the reference's LDPCEncoder / LDPCDecoder, operators/ldpc/
// encoder.h:48-75 and decoder.h:28-87, take both from cuPHY).
//
// Graph structure (TS 38.212 5.3.2, both NR base graphs): block rows 0..3
// ("core") span the kb information columns and the four core parity columns
// kb..kb+3; every later row i has one more column, kb + i, as an identity
// block.  Block (i, j) with shift s is the Z x Z identity with its columns
// cyclically shifted right by s: row r has its one in column (r + s) mod Z.
// With the first mb rows of the graph (mb = parity nodes, the code rate):
//
// Encode (one CTA per code block, 32 check nodes per word): lambda_i =
// sum_j P^s_ij s_j over the core rows' information entries, the core parity
// p = B^-1 lambda (B the 4Z x 4Z core block, inverted over GF(2) on the host
// once; the inverse of a block of circulants has circulant blocks, so its
// rows 0, Z, 2Z, 3Z give it as shift lists), then each extension row's parity
// from the information and core parity columns.  Out: the (kb - 2 + mb) Z bits after
// the 2Z punctured systematic ones (cuPHY's puncture option, nrLDPCEncode).
//
// Decode (one CTA per pair of code blocks, thread z = check node z of the
// current layer, both blocks in the two halves of FP16 pairs): LLRs (FP16,
// positive = bit 0) into a __half2 array in shared memory with the graph's
// entries; the rows in order as layers; per check node and block:
// q_e = app - r_e (r_e the node's previous message to entry e, rebuilt from
// its compressed state), min1, min2 and the parity of the sign bits of q,
// then app = q_e + r'_e, r'_e = +-min(0.75 min, 256).  Rows
// of up to 20 entries keep q in registers (ldpc_node, a variant per two
// degrees up to 12).  FP16 is the reference decoder's precision (cuPHY), and
// the pairs halve the instructions per block; channel LLRs clamped to
// +-1024 and messages to +-256 keep every value finite for up to 32 passes.
// Within a layer the Z check nodes touch disjoint variables (a circulant is
// a permutation), so a layer needs one barrier.  The compressed state (the two
// message magnitudes, who takes the second, sign bits) per (layer, check node)
// lives in global memory, loaded two layers ahead.  Every step is one IEEE FP16 operation, so the
// results equal the float16 restatement bit for bit.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "ldpc.cuh"

namespace mb {
namespace {

constexpr uint32_t kMaxZ = 384;
constexpr uint32_t kMaxDeg = 27;   // sign bits per check node and block in its state
constexpr float kAlpha = 0.75f;    // min-sum normalisation
// FP16 range: channel LLRs are clamped to +-kLlrMax once and every message
// to +-kMsgMax; q and app stay exact sums (app = llr + the messages of the
// variable's rows, up to rounding), below 1024 + 46 * 256 = 12800 with at
// most 46 rows, and the rounding of two operations a row visit (at most 32
// each below 65504) adds at most 46 * 32 * 32 in kMaxIter passes: nothing
// overflows.  (Clamping q or app instead breaks that sum: a later row then
// removes more of its old message than app still holds, and signs flip.)
constexpr float kLlrMax = 1024.f;
constexpr float kMsgMax = 256.f;
constexpr uint32_t kMaxIter = 32;

// Encoder bit streams: 32-bit words, bit 0 of the stream the most significant
// of word 0 (the MSB-first bytes of info and codewords in word form).  The 32
// bits from stream position pos on (reads words pos / 32 and the next one):
__device__ __forceinline__ uint32_t bits_at(const uint32_t *x, uint32_t pos) {
  return __funnelshift_l(x[pos / 32 + 1], x[pos / 32], pos & 31);
}
// bits o, o + 1, ... (indices mod Z, o < Z) of the Z-bit column at stream
// position base: a circulant's 32 rows as one word
__device__ __forceinline__ uint32_t rot_bits(const uint32_t *x, uint32_t base, uint32_t o, uint32_t Z) {
  uint32_t v = bits_at(x, base + o);
  const uint32_t f = Z - o;  // bits up to the column's end
  if (f < 32) {              // wraps
    v = (v & ~(0xFFFFFFFFu >> f)) | (bits_at(x, base) >> f);
    // a column shorter than a word repeats: its Z bits doubled (320 blocks of
    // 8 rows at Z = 2: 11.6 us with a wrap at a time, 8.0 so)
    if (Z < 32) {
      v &= ~(0xFFFFFFFFu >> Z);
      for (uint32_t n = Z; n < 32; n *= 2) v |= v >> n;
    }
  }
  return v;
}
// the first n bits (n >= 1) of v
__device__ __forceinline__ uint32_t first_bits(uint32_t v, uint32_t n) {
  return n >= 32 ? v : v & ~(0xFFFFFFFFu >> n);
}
// v (the bits past a column's end cleared) into the stream at position pos;
// neighbouring columns share words when Z % 32 != 0
__device__ __forceinline__ void put_bits(uint32_t *x, uint32_t pos, uint32_t v) {
  const uint32_t sh = pos & 31;
  if (v >> sh) atomicOr(x + pos / 32, v >> sh);
  if (sh && v << (32 - sh)) atomicOr(x + pos / 32 + 1, v << (32 - sh));
}

constexpr uint32_t kEncThreads = 512;

// One CTA per code block, the codeword's bit stream in shared memory, 32
// check nodes of a block row per thread: an entry costs one or two funnel
// shifts and an exclusive or for 32 rows.  Latency bound (five phases between
// barriers, a few KB in and out per block).  The core parity comes from
// B^-1, whose 4 x 4 blocks are sums of circulants like B's own (a few each
// for the standard's dual-diagonal core), applied entry by entry.  The first
// two products split an item's entries over four lanes: only 4 ceil(Z / 32)
// items exist.  320 blocks of base graph 1's shape at Z = 352: 161 us with a
// byte per bit and B^-1 as 4Z dense bit rows (62,000 words of B^-1 read per
// block), 9.8 us in this form.
__global__ void __launch_bounds__(kEncThreads) ldpc_encode_kernel(mb_ldpc h, const uint8_t *info,
                                                                  uint64_t info_stride, uint8_t *cw,
                                                                  uint64_t cw_stride) {
  extern __shared__ uint32_t enc_smem[];
  pdl_wait();
  const uint32_t Z = h.Z, kb = h.kb, mb = h.mb, tid = threadIdx.x, nt = blockDim.x;
  const uint32_t nw = (Z + 31) / 32;                // words per block of Z bits
  const uint32_t nx = ((kb + mb) * Z + 31) / 32 + 2;
  uint32_t *x = enc_smem;                           // the codeword, punctured bits included
  uint32_t *lam = x + nx;                           // lambda: four blocks of nw words, and one past them
  const uint8_t *in = info + (uint64_t)blockIdx.x * info_stride;
  const uint32_t in_bits = kb * Z, in_bytes = (in_bits + 7) / 8;
  const bool in_al = (reinterpret_cast<uintptr_t>(in) & 3) == 0;
  for (uint32_t w = tid; w < nx; w += nt) {
    uint32_t v = 0;
    if (in_al && 4 * w + 4 <= in_bytes) {
      v = __byte_perm(reinterpret_cast<const uint32_t *>(in)[w], 0, 0x0123);
    } else {
      for (uint32_t b = 4 * w; b < 4 * w + 4; b++) v = (v << 8) | (b < in_bytes ? in[b] : 0u);
    }
    x[w] = 32 * w < in_bits ? first_bits(v, in_bits - 32 * w) : 0u;
  }
  if (tid == 0) lam[4 * nw] = 0;
  __syncthreads();
  const uint32_t part = tid & 3, t4 = (4 * nw * 4 + 31) / 32 * 32;
  // lambda: the core rows over the information columns
  for (uint32_t t = tid; t < t4; t += nt) {
    const uint32_t i = t / 4 / nw, w = t / 4 % nw;
    uint32_t acc = 0;
    if (i < 4)
      for (uint32_t e = h.row_ptr[i] + part; e < h.row_ptr[i + 1]; e += 4) {
        const uint32_t c = h.col[e], o = 32 * w + h.sh[e];
        if (c < kb) acc ^= rot_bits(x, c * Z, o < Z ? o : o - Z, Z);
      }
    acc ^= __shfl_xor_sync(0xffffffffu, acc, 1);
    acc ^= __shfl_xor_sync(0xffffffffu, acc, 2);
    if (i < 4 && part == 0) lam[i * nw + w] = first_bits(acc, Z - 32 * w);
  }
  __syncthreads();
  // core parity p = B^-1 lambda
  for (uint32_t t = tid; t < t4; t += nt) {
    const uint32_t i = t / 4 / nw, w = t / 4 % nw;
    uint32_t acc = 0;
    if (i < 4)
      for (uint32_t e = __ldg(h.inv + i) + part, end = __ldg(h.inv + i + 1); e < end; e += 4) {
        const uint32_t en = __ldg(h.inv + e), o = 32 * w + (en & 0xFFFFu);
        acc ^= rot_bits(lam, (en >> 16) * nw * 32, o < Z ? o : o - Z, Z);
      }
    acc ^= __shfl_xor_sync(0xffffffffu, acc, 1);
    acc ^= __shfl_xor_sync(0xffffffffu, acc, 2);
    if (i < 4 && part == 0) put_bits(x, (kb + i) * Z + 32 * w, first_bits(acc, Z - 32 * w));
  }
  __syncthreads();
  // extension rows: one parity block each, from the information and core
  // parity columns (every other column's bits are still being written)
  for (uint32_t t = tid; t < (mb - 4) * nw; t += nt) {
    const uint32_t i = 4 + t / nw, w = t % nw;
    uint32_t acc = 0;
    for (uint32_t e = h.row_ptr[i]; e < h.row_ptr[i + 1]; e++) {
      const uint32_t c = h.col[e], o = 32 * w + h.sh[e];
      if (c < kb + 4) acc ^= rot_bits(x, c * Z, o < Z ? o : o - Z, Z);
    }
    put_bits(x, (kb + i) * Z + 32 * w, first_bits(acc, Z - 32 * w));
  }
  __syncthreads();
  // the encoded bits after the 2Z punctured ones, MSB first
  uint8_t *out = cw + (uint64_t)blockIdx.x * cw_stride;
  const uint32_t n_out = (kb - 2 + mb) * Z, out_bytes = (n_out + 7) / 8;
  const bool out_al = (reinterpret_cast<uintptr_t>(out) & 3) == 0;
  for (uint32_t w = tid; 4 * w < out_bytes; w += nt) {
    const uint32_t v = first_bits(bits_at(x, 2 * Z + 32 * w), n_out - 32 * w);
    if (out_al && 4 * w + 4 <= out_bytes) {
      reinterpret_cast<uint32_t *>(out)[w] = __byte_perm(v, 0, 0x0123);
    } else {
      for (uint32_t b = 0; b < 4 && 4 * w + b < out_bytes; b++) out[4 * w + b] = (uint8_t)(v >> (24 - 8 * b));
    }
  }
}

// Packed pairs: a CTA decodes two code blocks at once, lane 0 (the low half
// of every __half2) the pair's first block and lane 1 its second.
__device__ __forceinline__ uint32_t h2u(__half2 v) {
  uint32_t u;
  memcpy(&u, &v, 4);
  return u;
}
__device__ __forceinline__ __half2 u2h(uint32_t u) {
  __half2 v;
  memcpy(&v, &u, 4);
  return v;
}
__device__ __forceinline__ __half2 llr_clamp(__half2 v) {
  return __hmax2(__hmin2(v, __float2half2_rn(kLlrMax)), __float2half2_rn(-kLlrMax));
}

// A check node's state for the pair (one uint4 per layer and node) holds its
// messages: x, y the magnitudes min(0.75 min1, kMsgMax) and min(0.75 min2,
// kMsgMax) (__half2), z the message signs of entries 0..15 (bit e block 0, bit
// 16 + e block 1), and w
//   rows of at most kShortDeg entries: which entries take y (the |q| = min1
//     ones, in the layout of z);
//   longer rows: the signs of entries 16..26 in bits 0..10 / 16..26, and the
//     index of one |q| = min1 entry of block 0 in bits 11..15, of block 1 in
//     bits 27..31.
// Where several entries tie at min1, min2 = min1 and x = y, so neither form
// has to tell them apart.  The interleaving puts both blocks' bits for entry e
// at the same distance from bits 15 and 31, so one shift lines them up with
// the FP16 sign bits.
constexpr uint32_t kShortDeg = 12;
// bits 15 / 31 spread over their halves (byte permute with the selector's
// sign-replicate bit: bytes 1 and 3's top bits)
__device__ __forceinline__ uint32_t half_mask(uint32_t v) {
  uint32_t m;
  asm("prmt.b32 %0, %1, %2, 0xBB99;" : "=r"(m) : "r"(v), "r"(0u));
  return m;
}
// the message to entry j: z / w's bits for j in sg / y2 (w's for j >= 16)
__device__ __forceinline__ __half2 old_msg(uint32_t m1, uint32_t m2, uint32_t sg, uint32_t y2, uint32_t j) {
  const uint32_t sh = j < 16 ? 15 - j : 31 - j, sel = half_mask(y2 << sh);
  const uint32_t mag = (m1 & ~sel) | (m2 & sel);
  return u2h(mag ^ ((sg << sh) & 0x80008000u));
}
// a longer row's |q| = min1 indices as bits in the layout of z (entries 0..15)
// and of w's signs (16..26)
__device__ __forceinline__ void pos_bits(uint32_t w, uint32_t &lo, uint32_t &hi) {
  const uint32_t p0 = (w >> 11) & 31u, p1 = w >> 27;
  lo = (p0 < 16 ? 1u << p0 : 0u) | (p1 < 16 ? 1u << (16 + p1) : 0u);
  hi = (p0 >= 16 ? 1u << (p0 - 16) : 0u) | (p1 >= 16 ? 1u << p1 : 0u);
}
// the least and second least |q| so far and the signs' parity (bits 15, 31)
struct PairMin {
  __half2 min1, min2;
  uint32_t par;
  __device__ __forceinline__ void init() {
    min1 = min2 = __float2half2_rn(INFINITY);
    par = 0;
  }
  __device__ __forceinline__ void add(__half2 q) {
    const __half2 mag = u2h(h2u(q) & 0x7FFF7FFFu);
    min2 = __hmin2(min2, __hmax2(min1, mag));
    min1 = __hmin2(min1, mag);
    par ^= h2u(q);
  }
};
// the new messages and state of a row
struct PairNew {
  uint32_t m1, m2, sg, w;
  __device__ __forceinline__ void init(const PairMin &t, uint32_t deg) {
    const __half2 a = __float2half2_rn(kAlpha);  // 0.75, exact in FP16
    const __half2 cap = __float2half2_rn(kMsgMax);
    m1 = h2u(__hmin2(__hmul2(a, t.min1), cap));
    m2 = deg == 1 ? m1 : h2u(__hmin2(__hmul2(a, t.min2), cap));
    sg = w = 0;
  }
  // app = q + the message to entry j; SHORT: the short rows' state
  template <bool SHORT>
  __device__ __forceinline__ __half2 add(__half2 q, const PairMin &t, uint32_t j) {
    const uint32_t qb = h2u(q), sel = __heq2_mask(u2h(qb & 0x7FFF7FFFu), t.min1);
    const uint32_t sign = (qb ^ t.par) & 0x80008000u;
    if (SHORT || j < 16) sg |= sign >> (15 - j);
    else w |= sign >> (31 - j);
    if (SHORT) {
      w |= sel & (0x00010001u << j);
    } else {
      const uint32_t idx = sel & 0xF800F800u;  // the index fields: bits 11..15, 27..31
      w = (w & ~idx) | (j * 0x08000800u & idx);
    }
    return __hadd2(q, u2h(((m1 & ~sel) | (m2 & sel)) | sign));
  }
  __device__ __forceinline__ uint4 state() const { return make_uint4(m1, m2, sg, w); }
};
// entry en's slot of check node z (tid4 = 4 z): the variables wrap at Z
__device__ __forceinline__ __half2 *app_slot(uint8_t *app, const uint2 &en, uint32_t tid, uint32_t Z4) {
  return reinterpret_cast<__half2 *>(app + (en.x + 4 * tid - (tid >= en.y ? Z4 : 0u)));
}

// One check node's update for the pair over a row of MIN to D entries, all in
// registers: every app load issued before any store (a row holds one
// circulant per column block, so the node's D slots are distinct), then
// q_e = app - r_e (r_e from the node's previous state) with the min tracking,
// then app = q_e + r'_e.  Returns the new state.  The entries up to MIN need no
// look at the degree.
template <int MIN, int D>
__device__ __forceinline__ uint4 ldpc_node(uint8_t *app, const uint2 *ent, uint32_t deg, uint32_t tid, uint32_t Z4,
                                           const uint4 &st) {
  constexpr bool kShort = D <= (int)kShortDeg;
  // longer rows recompute the slots for the stores rather than hold them
  // (register pressure)
  __half2 *slot[kShort ? D : 1];
  __half2 q[D];
#pragma unroll
  for (int j = 0; j < D; j++) {
    if (j < MIN || j < (int)deg) {
      __half2 *a = app_slot(app, ent[j], tid, Z4);
      if constexpr (kShort) slot[j] = a;
      q[j] = *a;
    }
  }
  uint32_t y_lo = st.w, y_hi = 0;
  if constexpr (!kShort) pos_bits(st.w, y_lo, y_hi);
  PairMin t;
  t.init();
#pragma unroll
  for (int j = 0; j < D; j++) {
    if (j < MIN || j < (int)deg) {
      q[j] = __hsub2(q[j], old_msg(st.x, st.y, j < 16 ? st.z : st.w, j < 16 ? y_lo : y_hi, j));
      t.add(q[j]);
    }
  }
  PairNew n;
  n.init(t, deg);
#pragma unroll
  for (int j = 0; j < D; j++) {
    if (j < MIN || j < (int)deg) {
      __half2 *a;
      if constexpr (kShort) a = slot[j];
      else a = app_slot(app, ent[j], tid, Z4);
      *a = n.template add<kShort>(q[j], t, j);
    }
  }
  return n.state();
}

// The same update for rows of any degree (up to kMaxDeg): q_e is stored in
// place of app between the two passes.
__device__ __forceinline__ uint4 ldpc_node_any(uint8_t *app, const uint2 *ent, uint32_t deg, uint32_t tid,
                                               uint32_t Z4, const uint4 &st) {
  uint32_t y_lo, y_hi;
  pos_bits(st.w, y_lo, y_hi);
  PairMin t;
  t.init();
  for (uint32_t e = 0; e < deg; e++) {
    __half2 *a = app_slot(app, ent[e], tid, Z4);
    const __half2 qe = __hsub2(*a, old_msg(st.x, st.y, e < 16 ? st.z : st.w, e < 16 ? y_lo : y_hi, e));
    *a = qe;
    t.add(qe);
  }
  PairNew n;
  n.init(t, deg);
  for (uint32_t e = 0; e < deg; e++) {
    __half2 *a = app_slot(app, ent[e], tid, Z4);
    *a = n.add<false>(*a, t, e);
  }
  return n.state();
}

// CTA p decodes code blocks b0 + 2p and b0 + 2p + 1 (the second only when
// 2p + 1 < nb; otherwise its lane repeats the first and is not written)
__global__ void __launch_bounds__(kMaxZ, 2) ldpc_decode_kernel(mb_ldpc h, const __half *llr, uint64_t llr_stride,
                                                               uint8_t *out, uint64_t out_stride, uint32_t max_iter,
                                                               uint32_t b0, uint32_t nb) {
  // the pair's a-posteriori LLRs [(kb + mb) Z] (__half2), then the entries
  // {col * Z, shift} and the row pointers
  extern __shared__ uint32_t dec_smem[];
  pdl_wait();
  const uint32_t Z = h.Z, kb = h.kb, mb = h.mb, N = (kb + mb) * Z, tid = threadIdx.x, nt = blockDim.x;
  __half2 *app = reinterpret_cast<__half2 *>(dec_smem);
  uint2 *ent = reinterpret_cast<uint2 *>(dec_smem + (N + 1) / 2 * 2);  // [nnz]
  uint32_t *row = reinterpret_cast<uint32_t *>(ent + h.nnz);           // [mb]
  const uint32_t cb = b0 + 2 * blockIdx.x;
  const bool two = 2 * blockIdx.x + 1 < nb;
  const __half *in0 = llr + (uint64_t)cb * llr_stride;
  const __half *in1 = two ? in0 + llr_stride : in0;
  for (uint32_t v = tid; v < N; v += nt) app[v] = llr_clamp(__halves2half2(in0[v], in1[v]));
  // entry e as {4 (col * Z + shift), Z - shift}: check node z meets variable
  // col * Z + (z + shift) mod Z, at byte x + 4 z, less 4 Z once z >= y
  for (uint32_t e = tid; e < h.nnz; e += nt)
    ent[e] = make_uint2(4 * ((uint32_t)h.col[e] * Z + h.sh[e]), Z - h.sh[e]);
  uint8_t *appb = reinterpret_cast<uint8_t *>(app);
  const uint32_t Z4 = 4 * Z;
  // row i: first entry, degree in the upper half (27 entries of 8 bytes a row
  // at most: the shared memory ends long before 2^16 of them)
  for (uint32_t i = tid; i < mb; i += nt) row[i] = h.row_ptr[i] | (h.row_ptr[i + 1] - h.row_ptr[i]) << 16;
  __syncthreads();
  // Thread z only ever reads and writes check node z's state, so its loads
  // run two layers ahead of their use (a row's state is rewritten mb >= 4
  // layers before it is read again); the first pass starts from zero
  // messages without reading.
  uint4 *state = h.state + (uint64_t)blockIdx.x * mb * Z;
  const uint32_t layers = max_iter * mb;
  uint4 st_a = make_uint4(0u, 0u, 0u, 0u), st_b = st_a;
  uint32_t i = 0, i2 = 2, o = tid, o2 = 2 * Z + tid;  // this layer's row and the one two layers on, their state
  for (uint32_t l = 0; l < layers; l++) {
    const uint4 st = st_a;
    st_a = st_b;
    if (tid < Z) {
      if (l + 2 >= mb && l + 2 < layers) st_b = state[o2];
      const uint32_t rw = row[i], deg = rw >> 16;
      const uint2 *en = ent + (rw & 0xFFFFu);
      // every thread of the layer takes the same branch
      uint4 ns;
      if (deg <= 6) {
        if (deg <= 2)
          ns = ldpc_node<1, 2>(appb, en, deg, tid, Z4, st);
        else if (deg <= 4)
          ns = ldpc_node<3, 4>(appb, en, deg, tid, Z4, st);
        else
          ns = ldpc_node<5, 6>(appb, en, deg, tid, Z4, st);
      } else if (deg <= 10) {
        if (deg <= 8)
          ns = ldpc_node<7, 8>(appb, en, deg, tid, Z4, st);
        else
          ns = ldpc_node<9, 10>(appb, en, deg, tid, Z4, st);
      } else if (deg <= 12) {
        ns = ldpc_node<11, 12>(appb, en, deg, tid, Z4, st);
      } else if (deg <= 20) {
        ns = ldpc_node<13, 20>(appb, en, deg, tid, Z4, st);
      } else {
        ns = ldpc_node_any(appb, en, deg, tid, Z4, st);
      }
      state[o] = ns;
    }
    o += Z;
    o2 += Z;
    if (++i == mb) {
      i = 0;
      o = tid;
    }
    if (++i2 == mb) {
      i2 = 0;
      o2 = tid;
    }
    __syncthreads();
  }
  // hard decisions of the information bits, MSB first, both blocks
  uint8_t *o0 = out + (uint64_t)cb * out_stride, *o1 = o0 + out_stride;
  for (uint32_t b = tid; b < (kb * Z + 7) / 8; b += nt) {
    uint32_t v0 = 0, v1 = 0;
    for (uint32_t k = 0; k < 8; k++) {
      const uint32_t bit = 8 * b + k;
      const uint32_t ng = bit < kb * Z ? __hlt2_mask(app[bit], __float2half2_rn(0.f)) : 0u;
      v0 = (v0 << 1) | (ng & 1u);
      v1 = (v1 << 1) | (ng >> 31);
    }
    o0[b] = (uint8_t)v0;
    if (two) o1[b] = (uint8_t)v1;
  }
}

// B^-1 over GF(2) of the 4Z x 4Z core block, rows as 64-bit words; false
// when B is singular
bool core_inverse(const std::vector<std::vector<std::pair<uint32_t, uint32_t>>> &rows, uint32_t kb, uint32_t Z,
                  std::vector<uint64_t> &inv, uint32_t &w64) {
  const uint32_t n = 4 * Z;
  w64 = (n + 63) / 64;
  std::vector<uint64_t> a((size_t)n * w64, 0), b((size_t)n * w64, 0);
  for (uint32_t i = 0; i < 4; i++)
    for (auto &cs : rows[i])
      if (cs.first >= kb && cs.first < kb + 4)
        for (uint32_t r = 0; r < Z; r++) {
          const uint32_t c = (cs.first - kb) * Z + (r + cs.second) % Z;
          a[(size_t)(i * Z + r) * w64 + c / 64] ^= 1ull << (c % 64);
        }
  for (uint32_t r = 0; r < n; r++) b[(size_t)r * w64 + r / 64] = 1ull << (r % 64);
  for (uint32_t c = 0; c < n; c++) {
    uint32_t p = c;
    while (p < n && !((a[(size_t)p * w64 + c / 64] >> (c % 64)) & 1ull)) p++;
    if (p == n) return false;
    if (p != c)
      for (uint32_t w = 0; w < w64; w++) {
        std::swap(a[(size_t)p * w64 + w], a[(size_t)c * w64 + w]);
        std::swap(b[(size_t)p * w64 + w], b[(size_t)c * w64 + w]);
      }
    for (uint32_t r = 0; r < n; r++)
      if (r != c && ((a[(size_t)r * w64 + c / 64] >> (c % 64)) & 1ull))
        for (uint32_t w = 0; w < w64; w++) {
          a[(size_t)r * w64 + w] ^= a[(size_t)c * w64 + w];
          b[(size_t)r * w64 + w] ^= b[(size_t)c * w64 + w];
        }
  }
  inv.swap(b);
  return true;
}

}  // namespace
}  // namespace mb

using namespace mb;

extern "C" mb_status mb_ldpc_destroy(mb_ldpc *h) {
  if (!h) return MB_BAD_ARG;
  cudaFree(h->row_ptr);
  cudaFree(h->col);
  cudaFree(h->sh);
  cudaFree(h->inv);
  cudaFree(h->state);
  delete h;
  return MB_OK;
}

extern "C" mb_status mb_ldpc_create(const mb_ldpc_graph *g, uint32_t Z, uint32_t parity_nodes,
                                    uint32_t max_batch, mb_ldpc **out) {
  if (!g || !out || !g->row || !g->col || !g->shift) return MB_BAD_ARG;
  *out = nullptr;
  const uint32_t kb = g->kb, mbr = parity_nodes;
  if (Z == 0 || Z > kMaxZ || kb < 3 || mbr < 4 || mbr > g->rows || max_batch == 0) return MB_BAD_SHAPE;
  // rows < mb, entries by (row, col), shifts reduced mod Z (TS 38.212:
  // P = V mod Z); the NR block structure checked
  std::vector<std::vector<std::pair<uint32_t, uint32_t>>> rows(mbr);
  for (uint32_t k = 0; k < g->nnz; k++) {
    const uint32_t r = g->row[k], c = g->col[k];
    if (r >= g->rows || c >= kb + g->rows) return MB_BAD_ARG;
    if (r >= mbr) continue;
    const bool ext = c >= kb + 4;
    if (ext && (r < 4 || c != kb + r || g->shift[k] % Z != 0)) return MB_BAD_ARG;
    rows[r].push_back({c, (uint32_t)(g->shift[k] % Z)});
  }
  uint32_t nnz = 0;
  std::vector<uint32_t> row_ptr(mbr + 1, 0);
  std::vector<uint16_t> col, sh;
  for (uint32_t r = 0; r < mbr; r++) {
    std::sort(rows[r].begin(), rows[r].end());
    for (size_t k = 1; k < rows[r].size(); k++)
      if (rows[r][k].first == rows[r][k - 1].first) return MB_BAD_ARG;  // one circulant per block
    if (rows[r].empty() || rows[r].size() > kMaxDeg) return MB_BAD_ARG;
    if (r >= 4) {
      bool own = false;
      for (auto &cs : rows[r]) own |= cs.first == kb + r;
      if (!own) return MB_BAD_ARG;
    }
    for (auto &cs : rows[r]) {
      col.push_back((uint16_t)cs.first);
      sh.push_back((uint16_t)cs.second);
    }
    nnz += (uint32_t)rows[r].size();
    row_ptr[r + 1] = nnz;
  }
  std::vector<uint64_t> inv64;
  uint32_t w64 = 0;
  if (!core_inverse(rows, kb, Z, inv64, w64)) return MB_BAD_ARG;
  // block (i, j) of B^-1 is circulant: row i Z's ones at columns j Z + s give
  // its shifts s, entries (j << 16) | s
  std::vector<uint32_t> inv(5, 5);
  for (uint32_t i = 0; i < 4; i++) {
    for (uint32_t c = 0; c < 4 * Z; c++)
      if ((inv64[(size_t)i * Z * w64 + c / 64] >> (c % 64)) & 1ull) inv.push_back((c / Z) << 16 | c % Z);
    inv[i + 1] = (uint32_t)inv.size();
  }
  mb_ldpc *h = new mb_ldpc();
  h->kb = kb;
  h->Z = Z;
  h->mb = mbr;
  h->nnz = nnz;
  h->max_batch = max_batch;
  MB_CUDA_TRY(cudaGetDevice(&h->dev));
  mb_status st = MB_OK;
  auto alloc_copy = [&](void **p, const void *src, size_t bytes) {
    if (st != MB_OK) return;
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess && src) e = cudaMemcpy(*p, src, bytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) st = record_error(e);
  };
  alloc_copy((void **)&h->row_ptr, row_ptr.data(), row_ptr.size() * sizeof(uint32_t));
  alloc_copy((void **)&h->col, col.data(), col.size() * sizeof(uint16_t));
  alloc_copy((void **)&h->sh, sh.data(), sh.size() * sizeof(uint16_t));
  alloc_copy((void **)&h->inv, inv.data(), inv.size() * sizeof(uint32_t));
  alloc_copy((void **)&h->state, nullptr, (size_t)((max_batch + 1) / 2) * mbr * Z * sizeof(uint4));
  if (st != MB_OK) {
    mb_ldpc_destroy(h);
    return st;
  }
  *out = h;
  return MB_OK;
}

extern "C" mb_status mb_ldpc_encode(mb_ldpc *h, const uint8_t *info, uint64_t info_stride, uint8_t *cw,
                                    uint64_t cw_stride, uint32_t batch, void *stream) {
  if (!h || !info || !cw) return MB_BAD_ARG;
  if (info_stride < ((uint64_t)h->kb * h->Z + 7) / 8 ||
      cw_stride < ((uint64_t)(h->kb - 2 + h->mb) * h->Z + 7) / 8)
    return MB_BAD_SHAPE;
  if (batch == 0) return MB_OK;
  const size_t smem = 4 * (((size_t)(h->kb + h->mb) * h->Z + 31) / 32 + 2 + 4 * (size_t)((h->Z + 31) / 32) + 1);
  MB_CUDA_TRY(pdl_launch(ldpc_encode_kernel, batch, kEncThreads, smem, as_stream(stream), *h, info, info_stride, cw,
                         cw_stride));
  MB_LAUNCH_CHECK();
  return MB_OK;
}

extern "C" mb_status mb_ldpc_decode(mb_ldpc *h, const uint16_t *llr, uint64_t llr_stride, uint8_t *out,
                                    uint64_t out_stride, uint32_t batch, uint32_t max_iter, void *stream) {
  if (!h || !llr || !out) return MB_BAD_ARG;
  if (llr_stride < (uint64_t)(h->kb + h->mb) * h->Z || out_stride < ((uint64_t)h->kb * h->Z + 7) / 8)
    return MB_BAD_SHAPE;
  if (max_iter > kMaxIter) return MB_BAD_ARG;  // the FP16 range argument above
  if (batch == 0) return MB_OK;
  const size_t smem = ((size_t)(h->kb + h->mb) * h->Z + 1) / 2 * 8 + 8 * (size_t)h->nnz + 4 * ((size_t)h->mb + 1);
  static_assert(kMaxZ <= 1024, "one thread per check node");
  int maxs = 0;
  MB_CUDA_TRY(cudaDeviceGetAttribute(&maxs, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->dev));
  if (smem > (size_t)maxs) return MB_UNSUPPORTED;
  MB_CUDA_TRY(cudaFuncSetAttribute(ldpc_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const uint32_t threads = (h->Z + 31) / 32 * 32;
  // at most max_batch code blocks at a time, in pairs: each pair keeps its
  // check-node state
  for (uint32_t b0 = 0; b0 < batch; b0 += h->max_batch) {
    const uint32_t nb = std::min(h->max_batch, batch - b0);
    MB_CUDA_TRY(pdl_launch(ldpc_decode_kernel, (nb + 1) / 2, threads, smem, as_stream(stream), *h,
                           reinterpret_cast<const __half *>(llr), llr_stride, out, out_stride, max_iter, b0, nb));
    MB_LAUNCH_CHECK();
  }
  return MB_OK;
}
