// The whole-number arithmetic of a CTA's place in a launch: which row tile, head and batch it takes.  Host and device.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define AB200_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define AB200_HOST_DEVICE inline
#endif

namespace ab200 {

// a / b for 0 <= a, 0 < b by the fp32 reciprocal and corrections: at the start of a CTA every cycle of an integer division is waited for.
// Below 2^24 a is exact and the quotient at most one off, and so it is for quotients below 2^22.
AB200_HOST_DEVICE int reciprocal_quotient(int a, int b) {
#ifdef __CUDA_ARCH__
  return (int)((float)a * __frcp_rn((float)b));      // (2^31 becomes 2^31 - 1)
#else
  const float f = (float)a * (1.0f / (float)b);
  return f < 2147483648.0f ? (int)f : INT32_MAX;
#endif
}
// `a` below 2^24 or a quotient below 2^22
AB200_HOST_DEVICE int quick_div(int a, int b) {
  int q = reciprocal_quotient(a, b);
  int r = (int)((unsigned)a - (unsigned)q * (unsigned)b);
  if (r < 0) { --q; r += b; }
  if (r >= b) ++q;
  return q;
}
// Whatever they are: at 2^31 three roundings leave the first quotient a few hundred off.  (The loops, or an integer division beside it for
// large a, in place of quick_div's two corrections in the forward: 4 x 16:8 heads x 1000 causal of 128 42.2 -> 43.4 and 43.9 us.)
AB200_HOST_DEVICE int quick_div_any(int a, int b) {
  int q = reciprocal_quotient(a, b);
  int r = (int)((unsigned)a - (unsigned)q * (unsigned)b);
  while (r < 0) { --q; r += b; }
  while (r >= b) { ++q; r -= b; }
  return q;
}

// Which (row tile counted from the last, head, batch) the CTA (bx, by, bz) of an nx x nh x nz grid takes: heads in groups of 32, inside a group
// the row tiles slowest, so that the long tiles of a causal problem start together and first.  SNAKE: the CTAs that find room at once are
// dealt out a round of all SMs at a time, so every other round runs from the short tiles to the long ones; in the same order the SM with
// the longest first tile also had the longest second one.  Measured, forward, fp32, 2 x 8 x 500 x 64 causal: 35 -> 31 us.  (The backward's
// time is its longest CTA's, whichever SM that is on.)  32 bits count the CTAs: not for grids beyond_tile_order(), which the host gives to other
// kernels.  (A branch here instead, for every CTA: training step of 2 x 8 x 500 x 64 111.9 -> 113.7 us.)
constexpr int kTileHeadGroup = 32;
inline bool beyond_tile_order(int64_t nx, int64_t nh, int64_t nz) { return nx * nh * nz > INT32_MAX || nx > INT32_MAX / kTileHeadGroup; }
template <bool SNAKE>
AB200_HOST_DEVICE void tile_of_block(int bx, int by, int bz, int nx, int nh, int nz, int& x, int& h, int& z) {
  constexpr int kHeadGroup = kTileHeadGroup, kSms = 148;
  int lin = bx + nx * (by + nh * bz);
  if constexpr (SNAKE) {
    const int round = lin / kSms, round0 = round * kSms, rest = nx * nh * nz - round0;
    if (round & 1) lin = round0 + (rest < kSms ? rest : kSms) - 1 - (lin - round0);
  }
  const int grp = lin / (kHeadGroup * nx), r = lin - grp * (kHeadGroup * nx);
  const int left = nh * nz - grp * kHeadGroup, gsize = left < kHeadGroup ? left : kHeadGroup;
  x = r / gsize;
  const int hz = grp * kHeadGroup + (r - x * gsize);
  z = hz / nh;
  h = hz - z * nh;
}

}  // namespace ab200
