// A warp's 32 x 32 tile of bias or dBias (rows are queries, columns keys; 16-bit), between global memory and the two ways in which
// the tcgen05 kernels hold scores: a thread per row (forward, dQ) and a thread per column (dK/dV).
//
// In memory the tile is 32 rows of 64 bytes.  An access of a thread to its own row touches 32 lines, whatever its width, and
// occupies the load/store unit that often: 32-byte accesses (two a thread) halve it against 16-byte ones, and stores become
// full sectors.  A thread that reads its own column would need 32 2-byte loads; there four lanes share a row (lane 8q + e: columns
// 8q..8q+7 of rows 8t + e, t = 0..3, eight lines a load) and the lanes exchange.  Rows that are not aligned go that way too, element
// by element, all of a tile in flight.  (The exchange for aligned rows of the thread-per-row kernels as well: coalesced, but its
// shuffles and selects cost more than they save: forward of head dim 72 877 -> 1047 us, dQ 980 -> 1271.)
// Measured, device us, against 16-byte accesses to own rows, loaded behind the scores, and single elements where rows are not
// aligned: 8 x 16 heads x 2048, dropout 0.2: head dim 72 dQ 1139 -> 948, forward 895 -> 877; 256 dV 1787 -> 1443, dQ 1387 -> 1058,
// forward 1278 -> 1242; training step with bias alone, 4 x 16 x 1024 of 64, 335 -> 285; 2 x 16 x 1000 x 1001 of 128 835 -> 381;
// 2 x 4 x 300 of 160 211 -> 125.
#pragma once
#include "sm100_ptx.cuh"

namespace ab200 {

// `rows`, `cols`: what the matrix has from the tile's first row and column on (rows beyond repeat the last one, columns beyond are
// zero).  `vec`: rows are unit-stride and 16-byte aligned.  rs, cs: strides in elements.  (The choice is the warp's, not the
// lane's: the loads of one form stay in flight together.)
template <typename T>
__device__ __forceinline__ void tile32_load(uint4 (&raw)[4], const T* tile, int64_t rs, int64_t cs, bool vec, int rows, int cols, int lane) {
  const int q = lane >> 3, e = lane & 7;
  const uint16_t* base = reinterpret_cast<const uint16_t*>(tile) + 8 * q * cs;
  if (vec && cols >= 32) {
#pragma unroll
    for (int t = 0; t < 4; ++t) raw[t] = __ldg(reinterpret_cast<const uint4*>(base + (int64_t)min(8 * t + e, rows - 1) * rs));
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint16_t* src = base + (int64_t)min(8 * t + e, rows - 1) * rs;
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t lo = 8 * q + 2 * k < cols ? __ldg(src + 2 * k * cs) : 0, hi = 8 * q + 2 * k + 1 < cols ? __ldg(src + (2 * k + 1) * cs) : 0;
        w[k] = lo | hi << 16;
      }
      raw[t] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}
template <typename T>
__device__ __forceinline__ void tile32_store(const uint4 (&raw)[4], T* tile, int64_t rs, int64_t cs, bool vec, int rows, int cols, int lane) {
  const int q = lane >> 3, e = lane & 7;
  uint16_t* base = reinterpret_cast<uint16_t*>(tile) + 8 * q * cs;
  if (vec && cols >= 32) {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (8 * t + e < rows) *reinterpret_cast<uint4*>(base + (int64_t)(8 * t + e) * rs) = raw[t];
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (8 * t + e >= rows) continue;
      uint16_t* dst = base + (int64_t)(8 * t + e) * rs;
      const uint32_t w[4] = {raw[t].x, raw[t].y, raw[t].z, raw[t].w};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (8 * q + j < cols) dst[j * cs] = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
    }
  }
}
// A tile's rows towards L2, a lane a row: for the block after the one at hand.
template <typename T>
__device__ __forceinline__ void tile32_prefetch(const T* tile, int64_t rs, int64_t cs, int rows, int cols, int lane) {
  if (cols > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(tile + (int64_t)min(lane, rows - 1) * rs));
}
// Exchange between lane bits 3, 4 and the register index: from tile32_load's layout to the thread per row (lane l: raw[q] is columns
// 8q..8q+7 of row l) and back.
__device__ __forceinline__ void tile32_exchange(uint4 (&raw)[4], int lane) {
#pragma unroll
  for (int b = 1; b <= 2; b <<= 1) {
    const bool up = (lane & (8 * b)) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i & b) continue;
      uint4& lo = raw[i];
      uint4& hi = raw[i | b];
      const uint4 send = up ? lo : hi;
      uint4 got;
      got.x = __shfl_xor_sync(0xffffffffu, send.x, 8 * b);
      got.y = __shfl_xor_sync(0xffffffffu, send.y, 8 * b);
      got.z = __shfl_xor_sync(0xffffffffu, send.z, 8 * b);
      got.w = __shfl_xor_sync(0xffffffffu, send.w, 8 * b);
      if (up) lo = got; else hi = got;
    }
  }
}
// The thread per row: lane l has columns 8q..8q+7 of row l in raw[q].  Rows of 32-byte pieces (vec 2) take two 32-byte accesses a
// thread, full sectors each; with 16-byte pieces (vec 1) four.
template <typename T>
__device__ __forceinline__ void row32_load(uint4 (&raw)[4], const T* tile, int64_t rs, int64_t cs, int vec, int rows, int cols, int lane) {
  const T* src = tile + (int64_t)min(lane, rows - 1) * rs;
  if (vec == 2 && cols >= 32) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint4 &a = raw[2 * h], &b = raw[2 * h + 1];
      asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(src + 16 * h));
    }
  } else if (vec && cols >= 32) {
#pragma unroll
    for (int q = 0; q < 4; ++q) raw[q] = __ldg(reinterpret_cast<const uint4*>(src) + q);
  } else {
    tile32_load<T>(raw, tile, rs, cs, vec != 0, rows, cols, lane);
    tile32_exchange(raw, lane);
  }
}
template <typename T>
__device__ __forceinline__ void row32_store(uint4 (&raw)[4], T* tile, int64_t rs, int64_t cs, int vec, int rows, int cols, int lane) {
  T* dst = tile + (int64_t)lane * rs;
  if (vec == 2 && cols >= 32) {
    if (lane < rows) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 &a = raw[2 * h], &b = raw[2 * h + 1];
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(dst + 16 * h), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
      }
    }
  } else if (vec && cols >= 32) {
    if (lane < rows) {
#pragma unroll
      for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(dst)[q] = raw[q];
    }
  } else {
    tile32_exchange(raw, lane);
    tile32_store<T>(raw, tile, rs, cs, vec != 0, rows, cols, lane);
  }
}
// x[c] = x[c] * scale + bias[c] * log2(e) for the 32 columns of a thread per row: the products are rounded first, as the forward's
// reference point has them.
template <typename T>
__device__ __forceinline__ void add_bias_row32(float* x, const uint4 (&raw)[4], float scale) {
  const float2 s2 = make_float2(scale, scale), l2 = make_float2(kLog2e, kLog2e);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const T* b = reinterpret_cast<const T*>(&raw[q]);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const int c = 8 * q + j;
      const float2 r = ptx::fma2(make_float2(to_f32<T>(b[j]), to_f32<T>(b[j + 1])), l2, ptx::mul2(make_float2(x[c], x[c + 1]), s2));
      x[c] = r.x;
      x[c + 1] = r.y;
    }
  }
}
// The same for a thread per column (lane = key, x[c]: query row c of the tile), from tile32_load's layout: within each group of
// eight lanes an 8 x 8 transpose of 16-bit values, three exchange steps (lane bit <-> position bit).
template <typename T>
__device__ __forceinline__ void add_bias_column32(float* x, const uint4 (&raw)[4], float scale, int lane) {
  const float2 s2 = make_float2(scale, scale), l2 = make_float2(kLog2e, kLog2e);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    uint32_t w[4] = {raw[t].x, raw[t].y, raw[t].z, raw[t].w};
    // lane bit 0 <-> low/high half
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t o = __shfl_xor_sync(0xffffffffu, w[k], 1);
      w[k] = (lane & 1) ? __byte_perm(w[k], o, 0x3276) : __byte_perm(w[k], o, 0x5410);
    }
    // lane bit 1 <-> register index bit 0, lane bit 2 <-> register index bit 1
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
      const bool up = (lane & 2) != 0;
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? w[k] : w[k + 1], 2);
      if (up) w[k] = got; else w[k + 1] = got;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bool up = (lane & 4) != 0;
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? w[k] : w[k + 2], 4);
      if (up) w[k] = got; else w[k + 2] = got;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T* h = reinterpret_cast<const T*>(&w[k]);
      const int c = 8 * t + 2 * k;
      const float2 r = ptx::fma2(make_float2(to_f32<T>(h[0]), to_f32<T>(h[1])), l2, ptx::mul2(make_float2(x[c], x[c + 1]), s2));
      x[c] = r.x;
      x[c + 1] = r.y;
    }
  }
}

}  // namespace ab200
