// Device-side problem description and the arithmetic every attention kernel of
// this library shares: per-sequence geometry (dense / compact / padded / strided
// varlen), window parsing, the Philox dropout keep bit and dtype conversion.
//
// The formulas restate the behaviour of ROCm/aotriton's kernels:
//   sequence geometry   modules/flash/kernel/fwd_kernel.py:247-287
//   LSE / delta layout  modules/flash/kernel/fwd_kernel_inner.py:38-43
//   window parsing      modules/flash/kernel/masked_load_store.py:43-63
//   mask predicate      modules/flash/kernel/fwd_kernel_inner.py:127-150
//   dropout keep bit    modules/flash/kernel/dropout.py:16-70 (Philox4x32-10 as in
//                       triton/language/random.py:12-43)
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include "indexing.h"

namespace ab200 {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471824645996f;

// Every kernel's first statement.  Kernels are launched so that a grid may be set up while the one before it in the stream
// still runs (h_launch, cabi.cu): nothing may be read or written before this wait, which ends when all earlier grids have
// completed and their writes can be seen, and no thread may leave without it, or a later grid could overtake an earlier one.  The
// second instruction lets the next grid in the stream be set up in turn.
__device__ __forceinline__ void wait_for_earlier_grids() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct View4 {
  void* ptr;
  int64_t n[4];   // extents
  int64_t s[4];   // strides in elements
};

// Everything a kernel needs, passed by value as a __grid_constant__ parameter.
struct Params {
  View4 q, k, v, bias, out, dout, dq, dk, dv, dbias;
  float* lse;          // written by forward, read by backward
  float* delta;        // backward scratch
  int32_t batch, hq, hk, group;
  int32_t max_sq, max_sk, dqk, dvo;
  float sm_scale, qk_scale;       // qk_scale = sm_scale * log2(e)
  float dropout_p, dropout_scale; // dropout_scale = 1 / (1 - p)
  int32_t idropout;               // integer keep threshold
  int32_t dropout_on;
  int32_t causal;                 // causal_type != 0
  int32_t causal_type, window_left, window_right;
  int32_t varlen_mode;            // 0 dense, 1 compact/strided (THD), 2 padded (BHSD)
  const int32_t *cu_q, *cu_k, *ss_q, *ss_k;
  const uint64_t *seed_ptr, *off1_ptr;
  uint64_t off2;
  uint64_t *seed_out, *off_out;
  int32_t philox_head_offset, philox_hq;
  int32_t has_bias, has_dbias;
  int32_t bias_vec, dbias_vec;    // bias (dBias) rows are unit-stride and 16-byte (1), 32-byte (2) aligned, or not (0)
  uint32_t wait_limit_kcycles;    // bound of every in-kernel wait, in units of 1024 SM cycles (0 = about a second)
  int32_t drop_copy;              // test hook of the bounded waits: the producer leaves out one tile copy
                                  // (1 = first V block of the forward, 2 = first Q/dO block of dK/dV, 3 = first V block of dQ)
  int32_t packed_tiles;           // token-packed: the grid counts row tiles of all sequences instead of max_sq's per sequence
  int32_t hw_order;               // the forward's CTAs in the hardware's order: a grid of 2^24 or more, beyond quick_div
  unsigned int* ticket;           // dK/dV's ticket counter, zeroed by the preprocess kernel of the same call (null: by the launch itself)
  int32_t dk_from_db;             // dK = sm_scale * dBias^T Q, after the dQ kernel has written dBias (sm100_bwd_dk_db.cuh)
  int32_t keep_tiles, keep_shift; // keep bits of the first keep_tiles 32-key tiles pass through dQ's rows (0: none), or, with
                                  // keep_shift kKeepInDbias, through dBias; see KeepShare
};

// Geometry of one (sequence z) slice.
// What a tcgen05 kernel is compiled with.  At most 96 to 216 registers a thread go to the compute warps; what
// dropout (generator state, keep bits) and bias (its tile, pointers, strides) need is spilled around every block even where a
// call uses neither, so each combination has instantiations of its own.  kAll leaves everything to the run time (dBias without
// bias too).
enum : int { kPlain = 0, kBias = 1, kDropout = 2, kAll = 3 };      // bias, and its gradient or not; dropout; anything
inline int features(const Params& p) {
  if (p.has_dbias && !p.has_bias) return kAll;
  return (p.has_bias ? kBias : 0) | (p.dropout_on ? kDropout : 0);
}

struct Seq {
  int32_t sq, sk;        // actual lengths
  int64_t q0, k0;        // first token along the sequence axis
  int32_t bidx;          // index along the batch axis of the tensors
  int64_t lse_row;       // lse offset is (bidx*Hq + h) * lse_row + q0 + m
  int32_t wl, wr;        // parsed window (only meaningful when causal)
};

// `ends`: the cumulative lengths around sequence z (x, y queries, z, w keys); unused where the problem is dense.
__device__ __forceinline__ Seq seq_from_ends(const Params& p, int z, int4 ends) {
  Seq s;
  if (p.varlen_mode == 0) {
    s.sq = p.max_sq; s.sk = p.max_sk; s.q0 = 0; s.k0 = 0; s.bidx = z; s.lse_row = p.max_sq;
  } else {
    const int q_lo = ends.x, q_hi = ends.y, k_lo = ends.z, k_hi = ends.w;
    s.sq = q_hi - q_lo;
    s.sk = k_hi - k_lo;
    if (p.varlen_mode == 2) {          // padded: rank-4 tensors, lengths from cu_seqlens
      s.q0 = 0; s.k0 = 0; s.bidx = z; s.lse_row = p.max_sq;
    } else if (p.ss_q != nullptr) {    // strided THD: offsets from seq_strides
      s.q0 = p.ss_q[z]; s.k0 = p.ss_k[z]; s.bidx = 0; s.lse_row = p.ss_q[p.batch];
    } else {                           // compact THD
      s.q0 = q_lo; s.k0 = k_lo; s.bidx = 0; s.lse_row = p.cu_q[p.batch];
    }
  }
  const int32_t kTopLeft = -2147483647, kBottomRight = -2147483646;
  if (p.causal_type == 1 || p.window_left == kTopLeft) s.wl = s.sq;
  else if (p.causal_type == 2 || p.window_left == kBottomRight) s.wl = s.sq;
  else s.wl = p.window_left;
  if (p.causal_type == 1 || p.window_right == kTopLeft) s.wr = 0;
  else if (p.causal_type == 2 || p.window_right == kBottomRight) s.wr = s.sk - s.sq;
  else s.wr = p.window_right;
  return s;
}

__device__ __forceinline__ Seq resolve_seq(const Params& p, int z) {
  int4 ends = make_int4(0, 0, 0, 0);
  if (p.varlen_mode != 0) ends = make_int4(p.cu_q[z], p.cu_q[z + 1], p.cu_k[z], p.cu_k[z + 1]);
  return seq_from_ends(p, z, ends);
}

// Row tile `tile` of a token-packed batch, when the tiles of all sequences are counted through (within a
// sequence the last rows, which a causal mask lets see the most keys, come first).  A grid of max_sq's tiles
// for every sequence starts a CTA for each tile a shorter sequence does not have: at one CTA per SM each of
// them takes its turn.  Sequences are looked at 32 at a time by the whole warp, which hands on what it has read of the one it
// finds (`ends`).  False: beyond the last tile.
// Measured: 24 packed prompts of 32 to 2048 tokens, 32:8 heads of 128, 399 -> 372 us.
template <int ROWS>
__device__ __forceinline__ bool packed_tile(const Params& p, int tile, int lane, int& z, int& m0, int4& ends) {
  const int cap = (p.max_sq + ROWS - 1) / ROWS;      // a sequence longer than max_sq has no more tiles than that
  int before = 0;
  for (int b0 = 0; b0 < p.batch; b0 += 32) {
    int n = 0;
    int4 own = make_int4(0, 0, 0, 0);
    if (b0 + lane < p.batch) {
      own = make_int4(p.cu_q[b0 + lane], p.cu_q[b0 + lane + 1], p.cu_k[b0 + lane], p.cu_k[b0 + lane + 1]);
      n = max(0, min(cap, (own.y - own.x + ROWS - 1) / ROWS));
    }
    int upto = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const uint32_t past = __ballot_sync(0xffffffffu, before + upto > tile);
    if (past != 0u) {
      const int src = __ffs(past) - 1;
      z = b0 + src;
      m0 = (before + __shfl_sync(0xffffffffu, upto, src) - 1 - tile) * ROWS;
      ends = make_int4(__shfl_sync(0xffffffffu, own.x, src), __shfl_sync(0xffffffffu, own.y, src), __shfl_sync(0xffffffffu, own.z, src),
                       __shfl_sync(0xffffffffu, own.w, src));
      return true;
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}
// Upper bound of the number of tiles packed_tile() counts, from what the host knows: the packed token count.
// 0: not a batch for it (only consecutive sequences are bounded by that count; and past a few rounds of 32
// sequences the search costs a CTA more than the empty CTAs did: with the search for every count, 16:4 heads of 128,
// causal, 160 sequences of 16 to 400 tokens take 316 us instead of 299, 256 496 instead of 449, 4096 23.2 ms instead of
// 7.2; 160 of 32 to 2048 tokens the same, 256 2.81 ms instead of 2.76; 129 of them still gain, 1.47 -> 1.46).
inline int packed_tiles_bound(const Params& p, int rows) {
  if (p.varlen_mode != 1 || p.ss_q != nullptr || p.batch > 128) return 0;
  const int64_t per_seq = (int64_t)p.batch * ((p.max_sq + rows - 1) / rows);
  const int64_t by_tokens = p.q.n[2] / rows + p.batch;
  return by_tokens < per_seq ? (int)by_tokens : 0;
}

__device__ __forceinline__ int64_t lse_offset(const Params& p, const Seq& s, int h) {
  return ((int64_t)s.bidx * p.hq + h) * s.lse_row + s.q0;
}

// The elements of a warp's row segment (columns first..first + N - 1) that lie outside [lo, hi] become `fill`.  Where no row of the warp has
// a lower bound inside the segment (`no_lo`, warp-uniform: a causal mask, a sequence's end) one comparison an element is enough, with
// code for either.  ONE_BOUND false: two comparisons always, one piece of code.
// ONE_BOUND pays except beside bias and dropout together, where its second piece of code is spilled for around every block.  Measured, device us,
// two comparisons / one: forward, 4 x 16:8 heads x 2048 causal of 64 95.6 / 90.6, of 128 105.9 / 101.5; with bias and dropout, not causal, of 64
// 483.8 / 490.9, of 72 490 / 502 (1000 tokens of 64, which end inside a block, 151.6 / 149.2); dQ there, of 72, 556 / 577, of 128 548 / 577;
// dV of 256, in a whole backward, 1453 / 1462, but its dQ 703 / 696.  (To leave out of the forward's softmax the blocks that a warp sees nothing
// of costs registers as well: with one comparison, without and with it, of 128 101.5 / 103.2 causal, 164 / 170 not; bias and dropout of 72 490 / 546.)
template <int N, bool ONE_BOUND>
__device__ __forceinline__ void mask_columns(float* x, int first, int lo, int hi, bool no_lo, float fill) {
  if constexpr (ONE_BOUND) {
    lo -= first;
    hi -= first;
    if (no_lo) {
#pragma unroll
      for (int c = 0; c < N; ++c) x[c] = c <= hi ? x[c] : fill;
    } else {
#pragma unroll
      for (int c = 0; c < N; ++c) x[c] = (c >= lo && c <= hi) ? x[c] : fill;
    }
  } else {
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const int n = first + c;
      x[c] = (n >= lo && n <= hi) ? x[c] : fill;
    }
  }
}

// (m, n) relative to the sequence; true when the score takes part in the softmax.
__device__ __forceinline__ bool score_valid(const Params& p, const Seq& s, int m, int n) {
  bool ok = (m < s.sq) && (n < s.sk);
  if (p.causal) ok = ok && (n <= m + s.wr) && (n >= m - s.wl);
  return ok;
}

// Closed range of key indices that can be valid for query rows [m_lo, m_hi].
__device__ __forceinline__ void key_range(const Params& p, const Seq& s, int m_lo, int m_hi, int& n_lo, int& n_hi) {
  n_lo = 0; n_hi = s.sk - 1;
  if (p.causal) {
    int64_t lo = (int64_t)m_lo - s.wl, hi = (int64_t)m_hi + s.wr;
    if (lo > n_lo) n_lo = (int)(lo > 2147483647LL ? 2147483647LL : lo);
    if (hi < n_hi) n_hi = (int)(hi < -1 ? -1 : hi);
  }
}

// Closed range of query rows that can be valid for keys [n_lo, n_hi].
__device__ __forceinline__ void query_range(const Params& p, const Seq& s, int n_lo, int n_hi, int& m_lo, int& m_hi) {
  m_lo = 0; m_hi = s.sq - 1;
  if (p.causal) {
    int64_t lo = (int64_t)n_lo - s.wr, hi = (int64_t)n_hi + s.wl;
    if (lo > m_lo) m_lo = (int)(lo > 2147483647LL ? 2147483647LL : lo);
    if (hi < m_hi) m_hi = (int)(hi < -1 ? -1 : hi);
  }
}

// ---------------------------------------------------------------------------
// Philox4x32-10, counter = (offset lo, offset hi, 0, 0), key = (seed lo, seed hi).
struct Philox4 { uint32_t w[4]; };

__host__ __device__ __forceinline__ Philox4 philox4x32_10(uint64_t seed, uint64_t offset) {
  const uint32_t kA = 0xD2511F53u, kB = 0xCD9E8D57u, kKA = 0x9E3779B9u, kKB = 0xBB67AE85u;
  uint32_t c0 = (uint32_t)offset, c1 = (uint32_t)(offset >> 32), c2 = 0u, c3 = 0u;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    uint64_t pa = (uint64_t)kA * c0, pb = (uint64_t)kB * c2;
    uint32_t n0 = (uint32_t)(pb >> 32) ^ c1 ^ k0;
    uint32_t n2 = (uint32_t)(pa >> 32) ^ c3 ^ k1;
    c1 = (uint32_t)pb; c3 = (uint32_t)pa; c0 = n0; c2 = n2;
    k0 += kKA; k1 += kKB;
  }
  Philox4 r; r.w[0] = c0; r.w[1] = c1; r.w[2] = c2; r.w[3] = c3;
  return r;
}

// Dropout state of one (sequence, q-head): everything but the row/column part of the counter.
struct DropoutCtx {
  uint64_t seed, base;
  uint32_t stride;      // counters per row = ceil(max_seqlen_k / 4)
  int32_t threshold;
};

// `seed` and `offset` (= philox_offset1 + philox_offset2) as read from the device scalars: a kernel
// that walks several heads reads them once and builds each head's context from the values.
__device__ __forceinline__ DropoutCtx dropout_ctx_from(const Params& p, uint64_t seed, uint64_t offset, int z, int h) {
  DropoutCtx d;
  d.seed = seed;
  d.stride = (uint32_t)((p.max_sk + 3) / 4);
  int hq_total = p.philox_hq > 0 ? p.philox_hq : p.hq;
  uint64_t zh = (uint64_t)z * hq_total + (uint64_t)(h + p.philox_head_offset);
  d.base = offset + zh * (uint64_t)p.max_sq * d.stride;
  d.threshold = p.idropout;
  return d;
}

__device__ __forceinline__ DropoutCtx dropout_ctx(const Params& p, int z, int h) {
  return dropout_ctx_from(p, p.seed_ptr ? *p.seed_ptr : 0ull, p.off2 + (p.off1_ptr ? *p.off1_ptr : 0ull), z, h);
}

// The four 32-bit words of one counter serve columns 4c..4c+3 in the order w0, w2, w1, w3.
__device__ __forceinline__ uint32_t philox_word_for_column(const Philox4& r, int n) {
  int j = n & 3;
  return j == 0 ? r.w[0] : (j == 1 ? r.w[2] : (j == 2 ? r.w[1] : r.w[3]));
}

__device__ __forceinline__ bool dropout_keep(const DropoutCtx& d, int m, int n) {
  Philox4 r = philox4x32_10(d.seed, d.base + (uint64_t)m * d.stride + (uint64_t)(n >> 2));
  return (int32_t)philox_word_for_column(r, n) > d.threshold;
}

// Keep bits of columns 4c..4c+3 of row m as a 4-bit mask (bit j = column 4c+j).
__device__ __forceinline__ uint32_t dropout_keep4(const DropoutCtx& d, int m, int c) {
  Philox4 r = philox4x32_10(d.seed, d.base + (uint64_t)m * d.stride + (uint64_t)c);
  uint32_t k = 0;
  k |= ((int32_t)r.w[0] > d.threshold) ? 1u : 0u;
  k |= ((int32_t)r.w[2] > d.threshold) ? 2u : 0u;
  k |= ((int32_t)r.w[1] > d.threshold) ? 4u : 0u;
  k |= ((int32_t)r.w[3] > d.threshold) ? 8u : 0u;
  return k;
}

// N counters of one seed in lockstep: independent chains side by side, and the two key additions of a round
// serve all of them.  (Ten round keys held in registers save the additions too, but twenty registers is what the
// compute warps do not have: dK/dV with dropout, head dim 128, spilled 228 bytes with them, 156 without.  Measured, training step of 16
// packed sequences of 64 to 8192 tokens, 32:8 heads of 128, dropout 0.1: 22.73 -> 21.85 ms; bias, dropout 0.2,
// 8 x 16 heads x 2048: head dim 72 3.58 -> 3.52, 256 5.53 -> 5.38.  The halves of a product by separate
// instructions, which alone have less latency than the wide multiply, changed nothing here.)
// c[n][0..1]: counter in, words 0 and 1 out; c[n][2..3]: words 2 and 3 out.
template <int N>
__device__ __forceinline__ void philox4x32_10_lockstep(uint64_t seed, uint32_t (&c)[N][4]) {
  const uint32_t kA = 0xD2511F53u, kB = 0xCD9E8D57u, kKA = 0x9E3779B9u, kKB = 0xBB67AE85u;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  asm volatile("" : "+r"(k0), "+r"(k1));      // (the sums are formed here, not once and kept)
#pragma unroll
  for (int n = 0; n < N; ++n) c[n][2] = c[n][3] = 0u;
#pragma unroll
  for (int i = 0; i < 10; ++i) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const uint64_t pa = (uint64_t)kA * c[n][0], pb = (uint64_t)kB * c[n][2];
      const uint32_t n0 = (uint32_t)(pb >> 32) ^ c[n][1] ^ k0;
      const uint32_t n2 = (uint32_t)(pa >> 32) ^ c[n][3] ^ k1;
      c[n][1] = (uint32_t)pb; c[n][3] = (uint32_t)pa; c[n][0] = n0; c[n][2] = n2;
    }
    k0 += kKA; k1 += kKB;
  }
}

// Keep bits of one row (or key) and 32 columns: the bit of column 4a + b is bit 8b + 7 - a, so that the word shifted left by a
// has the bits of columns 4a..4a+3 as the signs of its bytes, which one byte permute spreads over a pair of 16-bit halves
// (keep_mask).  In the natural order a column took a test and a select of its own, for P and again for dP.  Measured, dK/dV and dQ on
// the device, ms (with the reads of dP in two halves, sm100_bwd.cu): 16 packed sequences of 64 to 8192 tokens, 32:8 heads of 128, 9.93 ->
// 8.98 and 5.54 -> 5.45; 8 x 16 heads x 2048 of 72 with bias 1.42 -> 1.31 and 1.145 -> 1.139; head dim 256, dV, 1.92 -> 1.79.
// keep_bits(): the bits of counters `first`..`first` + N - 1 of such a word, counter a being columns 4a..4a+3.  `offset(n)`: the
// n-th of them.
template <int N, typename F>
__device__ __forceinline__ uint32_t keep_bits(uint64_t seed, int32_t threshold, int first, F offset) {
  uint32_t c[N][4], k = 0u;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const uint64_t o = offset(n);
    c[n][0] = (uint32_t)o;
    c[n][1] = (uint32_t)(o >> 32);
  }
  philox4x32_10_lockstep<N>(seed, c);
#pragma unroll
  for (int n = 0; n < N; ++n) {
    k |= ((int32_t)c[n][0] > threshold) ? 1u << (7 - first - n) : 0u;
    k |= ((int32_t)c[n][2] > threshold) ? 1u << (15 - first - n) : 0u;
    k |= ((int32_t)c[n][1] > threshold) ? 1u << (23 - first - n) : 0u;
    k |= ((int32_t)c[n][3] > threshold) ? 1u << (31 - first - n) : 0u;
  }
  return k;
}
__device__ __forceinline__ int keep_bit_of(int column) { return 8 * (column & 3) + 7 - (column >> 2); }
__device__ __forceinline__ int keep_column_of(int bit) { return 4 * (7 - (bit & 7)) + (bit >> 3); }
// Columns 2 * pair and 2 * pair + 1 of a keep word: all ones in the halves of those that are kept.
__device__ __forceinline__ uint32_t keep_mask(uint32_t w, int pair) {
  uint32_t m;
  if (pair & 1) asm("prmt.b32 %0, %1, 0, 0xbbaa;" : "=r"(m) : "r"(w << (pair >> 1)));
  else asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(m) : "r"(w << (pair >> 1)));
  return m;
}

// ---------------------------------------------------------------------------
// KeepShare: keep bits drawn once per backward.  Philox bounds the dropout kernels (ten serial rounds
// per four scores), and dK/dV and dQ need the same bits.  When both run in one call, the kernel that
// runs first (dK/dV; dV for wide heads) leaves the bits it drew in rows of dQ that only the last kernel
// writes, and the later ones read them: one bit per score moved instead of ten Philox rounds per four.
// Unit: 32 query rows (aligned to 32 in the sequence) x 32 keys = 32 words, one per query row (keep_bits()).  The words of a tile are 128 contiguous bytes (one coalesced access of a warp) in one
// of the same 32 rows of dQ; a row takes 2^keep_shift tiles (its 2 * dqk bytes allow no more), so the 32 rows
// hold 32 << keep_shift key tiles: 1024 keys at head dims 64 to 127, 2048 up to 255, 4096 at 256.  Tiles
// further right, partial row groups and all other launches draw their bits.
// A CTA of the dQ kernel reads the words of its own 128 rows only, and writes these rows after its
// last block, so nothing is overwritten before it has been read.
// Measured, forward + backward before and after: head dim 256, bias, dropout 0.2, 8 x 16 heads x 2048 tokens 7.43 ->
// 6.74 ms (two of three draws gone); head dim 72 3.82 -> 3.77 (half of the keys have room); 16 packed sequences of
// 64 to 8192 tokens, 32:8 heads of 128, 23.41 -> 23.09; 16 x 12 heads x 391, head dim 64, 0.66 -> 0.65.
// Where dBias is written, each tile's words go into its own 32 x 32 of it, 64 bytes into the first row and 64 into the second:
// there is room for every whole tile of keys, and the warp of the dQ kernel that reads them is the one that then writes these
// 32 x 32.  Measured, 8 x 16 heads x 2048 of 72 with bias, dropout 0.2 (half of the keys have room in dQ): dQ 948 -> 832 us, dK/dV 1312 -> 1343 (all of its bits are stored).
// `row32`: first of the 32 query rows; `key0`: first key of the tile (both multiples of 32).  IN_DBIAS: compiled with dBias.
constexpr int kKeepInDbias = -1;
template <bool IN_DBIAS>
__device__ __forceinline__ uint32_t* keep_share_word(const Params& p, const Seq& sq, int h, int row32, int key0, int lane) {
  if (IN_DBIAS && p.keep_shift == kKeepInDbias) {
    char* base = reinterpret_cast<char*>(p.dbias.ptr) +
                 2 * ((int64_t)sq.bidx * p.dbias.s[0] + (int64_t)h * p.dbias.s[1] + (int64_t)(row32 + (lane >> 4)) * p.dbias.s[2] + key0);
    return reinterpret_cast<uint32_t*>(base) + (lane & 15);
  }
  const int t = key0 >> 5;
  const int64_t row = sq.q0 + row32 + (t >> p.keep_shift);
  char* base = reinterpret_cast<char*>(p.dq.ptr) +
               2 * ((int64_t)sq.bidx * p.dq.s[0] + (int64_t)h * p.dq.s[1] + row * p.dq.s[2]);
  return reinterpret_cast<uint32_t*>(base + ((t & ((1 << p.keep_shift) - 1)) << 7)) + lane;
}

// Writer and readers agree by this rule on the tiles whose bits are shared.  A tile in which every score
// is masked is left out: the kernels differ in which of those they visit at all.
__device__ __forceinline__ bool keep_shared(const Params& p, const Seq& sq, int row32, int key0) {
  if ((key0 >> 5) >= p.keep_tiles || row32 + 32 > min(sq.sq, p.max_sq)) return false;
  return !p.causal || ((int64_t)row32 + 31 + sq.wr >= key0 && (int64_t)row32 - sq.wl <= (int64_t)key0 + 31);
}

// Key-per-thread kernels: a counter serves four consecutive keys of one query row, and the four lanes of a quad own exactly such
// keys.  Lane 4a + q of a warp draws for query rows q + 4k (k = 0..7): byte j, bit 7 - k of `x` is key 4a + j.

// The bits of this lane's own key over the 32 query rows, as a keep word.
__device__ __forceinline__ uint32_t keep_word_of_key(uint32_t x, int lane) {
  const uint32_t sel = (uint32_t)(lane & 3) | (uint32_t)(4 + (lane & 3)) << 4;      // (the byte of this lane's key in either word)
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = __shfl_sync(0xffffffffu, x, (lane & ~3) | i);
  return __byte_perm(__byte_perm(w[0], w[1], sel), __byte_perm(w[2], w[3], sel), 0x5410);
}
// The writer's side: an 8 x 8 transpose of bits over the lanes with the same q, in each byte, gives lane l the keep word of query
// row l.  (Lane bit against bit index, which counts down: lane 4a + q, bit 7 - k goes to lane 4k + q, bit 7 - a.)
__device__ __forceinline__ uint32_t keep_rows_from_quads(uint32_t x, int lane) {
#pragma unroll
  for (int b = 1; b < 8; b <<= 1) {
    const uint32_t m = b == 1 ? 0xaaaaaaaau : (b == 2 ? 0xccccccccu : 0xf0f0f0f0u);
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4 * b);
    x = (lane & (4 * b)) ? ((x & ~m) | ((y & ~m) << b)) : ((x & m) | ((y & m) >> b));
  }
  return x;
}

// 32 x 32 bit transpose over the warp: lane l's bit c becomes lane c's bit l.
__device__ __forceinline__ uint32_t transpose_bits32(uint32_t x, int lane) {
#pragma unroll
  for (int b = 16; b > 0; b >>= 1) {
    const uint32_t m = b == 16 ? 0x0000ffffu : (b == 8 ? 0x00ff00ffu : (b == 4 ? 0x0f0f0f0fu : (b == 2 ? 0x33333333u : 0x55555555u)));
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, b);
    x = (lane & b) ? ((x & ~m) | ((y >> b) & m)) : ((x & m) | ((y << b) & ~m));
  }
  return x;
}
// A reader whose lanes are keys: lane l has the keep word of query row l and gets that of key l.
__device__ __forceinline__ uint32_t keep_keys_from_rows(uint32_t x, int lane) {
  x = __shfl_sync(0xffffffffu, x, keep_column_of(lane));      // (rows in the order of their bits)
  return __shfl_sync(0xffffffffu, transpose_bits32(x, lane), keep_bit_of(lane));
}

// ---------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// dBias of query rows [m0, m0 + rows) outside the key columns [c_lo, c_hi) that the calling CTA's
// block loop visits.  A causal or windowed problem skips whole key blocks; the gradient of the bias
// there is zero, and it is written, so that dBias is defined everywhere inside the sequence.  (The
// reference leaves those entries as they were: modules/flash/kernel/bwd_inner_dq.py:200-204 stores
// dB only in the blocks its loop visits.)  Called by all threads of the CTA.
template <typename T>
__device__ __forceinline__ void zero_dbias_outside(const Params& p, const Seq& sq, int h, int m0, int rows, int c_lo,
                                                   int c_hi) {
  if (!p.has_dbias || !p.causal) return;
  const int lane = threadIdx.x & 31, nwarps = (int)blockDim.x >> 5;
  for (int r = (int)threadIdx.x >> 5; r < rows; r += nwarps) {
    const int m = m0 + r;
    if (m >= sq.sq) break;
    T* rowp = reinterpret_cast<T*>(p.dbias.ptr) + (int64_t)sq.bidx * p.dbias.s[0] + (int64_t)h * p.dbias.s[1] +
              (int64_t)m * p.dbias.s[2];
    for (int n = lane; n < min(c_lo, sq.sk); n += 32) rowp[(int64_t)n * p.dbias.s[3]] = from_f32<T>(0.f);
    for (int n = max(c_hi, 0) + lane; n < sq.sk; n += 32) rowp[(int64_t)n * p.dbias.s[3]] = from_f32<T>(0.f);
  }
}

// Round through the storage type, the way the reference casts P and dS before its GEMMs.
template <typename T> __device__ __forceinline__ float round_to(float x) { return to_f32<T>(from_f32<T>(x)); }

}  // namespace ab200
