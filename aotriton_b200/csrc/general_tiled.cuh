// General attention kernels for head dims up to 128: register tiles on the fp32 arithmetic units.
// Included by general_kernels.cu inside its namespaces.
//
// What bounds them: 16-byte shared-memory reads (an 8-read step feeds 64 multiply-adds per thread) where the
// grid fills the chip, the latency of a block's chain -- stage, scores, softmax, accumulate -- where it does
// not.  The 16x16-tile kernels (kept for head dims above 128) compute one dot product per thread, two
// reads for every four multiply-adds.  Here 128 threads own 32 rows (queries; keys for
// dK / dV) and walk the other sequence dimension in blocks of BN columns; a thread holds a 4 x BN/16
// tile of scores (rows ty*4.., columns tx + 16 j) and a 4 x DP/16 tile of each accumulator (columns tx*4.. + 64 j),
// so that a 16-byte read feeds 8 or more multiply-adds.  32 rows and not 64: at the sizes single precision is
// used at, the number of CTAs is what is short.  fp32 tiles are copied asynchronously, a block ahead of their use
// where a tile's last reader is known early.  Measured, fp32, 2 x 8 heads x 500 tokens, head dim 64, causal, nothing in L2,
// against loads through registers with one group of warps a tile: forward 98 -> 35 us, backward 139 -> 110 (97 once the copy loops fit the instruction cache).
//
// All tiles are row-major fp32 with four floats of padding: (DP + 4) / 4 is odd, so the 16 lanes that
// read 16 different rows at one column hit different banks.  The P / dS rows that a warp writes are read
// back by that warp only.
template <int DP> struct Tiled {
  static constexpr int kThreads = 128, kBM = 32;
  static constexpr int kBN = DP > 64 ? 32 : 64;
  static constexpr int kNC = kBN / 16;        // score columns per thread
  static constexpr int kND = DP / 64;         // float4 accumulator columns per thread
  static constexpr int kLd = DP + 4, kLdP = kBN + 4;
};

// 16-byte (fp32) or 8-byte (16-bit types) loads of four elements are possible on every row of the view.
template <typename T>
__device__ __forceinline__ bool rows_vec4(const View4& v, int d) {
  return ((reinterpret_cast<uintptr_t>(v.ptr) & (4 * sizeof(T) - 1)) == 0) && ((v.s[0] | v.s[1] | v.s[2]) & 3) == 0 && (d & 3) == 0;
}

// A thread's part of a tile through registers: rows `kStep` apart, `rows` of them (from the first) in the tensor, `cols` of its four
// columns.
template <typename T, int DP, int ROWS, int kStep, int kUnroll>
__device__ __forceinline__ void stage_loaded(float* dst, const T* src, int64_t stride, int rows, int cols, bool vec) {
#pragma unroll kUnroll
  for (int i = 0; i < ROWS / kStep; ++i) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i * kStep < rows && cols > 0) {
      const T* s = src + (int64_t)(i * kStep) * stride;
      if (sizeof(T) == 2 && vec) {
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(s));
        const T* e = reinterpret_cast<const T*>(&w);
        x = make_float4(to_f32<T>(e[0]), to_f32<T>(e[1]), to_f32<T>(e[2]), to_f32<T>(e[3]));
      } else {
        x.x = to_f32<T>(s[0]);
        if (cols > 1) x.y = to_f32<T>(s[1]);
        if (cols > 2) x.z = to_f32<T>(s[2]);
        if (cols > 3) x.w = to_f32<T>(s[3]);
      }
    }
    *reinterpret_cast<float4*>(dst + i * kStep * Tiled<DP>::kLd) = x;
  }
}
// fp32 rows that cannot be copied 16 bytes at a time; out of line, so that the copies of aligned rows are all that the kernels' loops hold.
template <typename T, int DP, int ROWS, int kStep>
static __device__ __noinline__ void stage_elements(float* dst, const T* src, int64_t stride, int rows, int cols) {
  stage_loaded<T, DP, ROWS, kStep, 4>(dst, src, stride, rows, cols, false);
}

// Rows row0.. of one head into dst[ROWS][DP + 4]; rows at or beyond nrows and columns at or beyond d
// are zero (columns up to the next multiple of four: the contractions stop there, the accumulators' ones
// are never stored).  `tid` of THREADS threads.  fp32 rows that allow it are copied asynchronously, all of a tile in flight at
// once: stage_wait() and a barrier come before their use.  (Through registers four loads were in flight, and half of the
// forward's time went by waiting for them.)
template <typename T, int DP, int ROWS, int THREADS>
__device__ __forceinline__ void stage_tile(float* dst, const View4& v, int b, int h, int64_t tok0, int row0, int nrows, int d, bool vec, int tid) {
  constexpr int kLd = Tiled<DP>::kLd, kC4 = DP / 4, kStep = THREADS / kC4;      // a thread's column, rows kStep apart
  static_assert(THREADS % kC4 == 0 && ROWS % kStep == 0, "whole rows a pass");
  const int r0 = tid / kC4, c = (tid - r0 * kC4) * 4;
  const T* src = row_ptr<T>(v, b, h, tok0 + row0 + r0) + c;
  dst += r0 * kLd + c;
  // (rolled up where nothing is gained: the unrolled forms of all a kernel's tiles together did not fit the instruction cache)
  if constexpr (sizeof(T) == 4) {
    if (vec) {
      const int in = c < d ? nrows - row0 - r0 : 0;      // rows to copy from here on
      uint32_t to = ptx::smem_u32(dst);
      const int64_t step = kStep * v.s[2];
#pragma unroll 2
      for (int i = 0; i < ROWS; i += kStep, to += kStep * kLd * 4, src += step)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     ::"r"(to), "l"(i < in ? src : reinterpret_cast<const T*>(v.ptr)), "r"(i < in ? 16 : 0) : "memory");
    }
  }
  if (sizeof(T) != 4) {
    stage_loaded<T, DP, ROWS, kStep, 4>(dst, src, v.s[2], nrows - row0 - r0, c < d ? d - c : 0, vec);
  } else if (!vec) {
    stage_elements<T, DP, ROWS, kStep>(dst, src, v.s[2], nrows - row0 - r0, c < d ? d - c : 0);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// This thread's copies have landed, all but those of its last PENDING stage_tile calls.
template <int PENDING>
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// s[i][j] = A[ty*4 + i] . B[tx + 16 j] over d4 groups of four columns, even and odd columns in the two halves of a packed
// sum (two multiply-adds an instruction: the issue slots, not the arithmetic, are what a block of few warps is short of)
template <int DP>
__device__ __forceinline__ void tile_dots(float (&s)[4][Tiled<DP>::kNC], const float* A, const float* B, int d4, int ty, int tx) {
  using C = Tiled<DP>;
  float2 t[4][C::kNC];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < C::kNC; ++j) t[i][j] = make_float2(0.f, 0.f);
  const float* a0 = A + ty * 4 * C::kLd;
  const float* b0 = B + tx * C::kLd;
#pragma unroll 2
  for (int c = 0; c < d4; ++c) {
    float4 a[4], b[C::kNC];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(a0 + i * C::kLd + c * 4);
#pragma unroll
    for (int j = 0; j < C::kNC; ++j) b[j] = *reinterpret_cast<const float4*>(b0 + j * 16 * C::kLd + c * 4);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < C::kNC; ++j) {
        t[i][j] = ptx::fma2(make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y), t[i][j]);
        t[i][j] = ptx::fma2(make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w), t[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < C::kNC; ++j) s[i][j] = t[i][j].x + t[i][j].y;
}

// The part [k0, k1) of the block of BN columns at `col0` that some row of the warp's eight sees (columns lo..hi), k0
// rounded down to eight.  The accumulations stop there.  A masked pair's weight is zero, but zero times a non-finite row
// of X is not: a row must not depend on rows that neither it nor its neighbours in the warp see.  (The 16x16-tile
// kernels keep the same distance with their tiles.)
template <int DP>
__device__ __forceinline__ void seen_columns(int lo, int hi, int col0, int& k0, int& k1) {
  k0 = max(lo - col0, 0) & ~7;
  k1 = min(hi - col0 + 1, Tiled<DP>::kBN);
}
constexpr int kWarpRows = 8;      // rows of a tile whose weights one warp writes and reads

// acc[i][j] += P[ty*4 + i][k..k + 4) x X[k..k + 4)[tx*4 + 64 j ..]
template <int DP>
__device__ __forceinline__ void accumulate4(float4 (&acc)[4][Tiled<DP>::kND], const float* p0, const float* x0, int k) {
  using C = Tiled<DP>;
  float4 a[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(p0 + i * C::kLdP + k);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk)
#pragma unroll
    for (int j = 0; j < C::kND; ++j) {
      const float4 x = *reinterpret_cast<const float4*>(x0 + (k + kk) * C::kLd + 64 * j);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float w = kk == 0 ? a[i].x : (kk == 1 ? a[i].y : (kk == 2 ? a[i].z : a[i].w));
        acc[i][j].x = fmaf(w, x.x, acc[i][j].x);
        acc[i][j].y = fmaf(w, x.y, acc[i][j].y);
        acc[i][j].z = fmaf(w, x.z, acc[i][j].z);
        acc[i][j].w = fmaf(w, x.w, acc[i][j].w);
      }
    }
}

// The same over [k0, k1); k0 is a multiple of eight, k1 is rounded up to one.  (Pointers that advance, eight columns an
// iteration: measured like a loop over the whole block.  Indexed by k, or four columns at a time, the forward took up to
// 24 % more and the backward up to 4 %.)
template <int DP>
__device__ __forceinline__ void tile_accumulate(float4 (&acc)[4][Tiled<DP>::kND], const float* P, const float* X, int k0, int k1, int ty, int tx) {
  using C = Tiled<DP>;
  static_assert(C::kBN % 8 == 0, "a rounded-up k1 stays inside the block");
  const float* p0 = P + ty * 4 * C::kLdP + k0;
  const float* x0 = X + k0 * C::kLd + tx * 4;
#pragma unroll 1
  for (int n = (k1 - k0 + 7) >> 3; n > 0; --n) {
    accumulate4<DP>(acc, p0, x0, 0);
    accumulate4<DP>(acc, p0, x0, 4);
    p0 += 8;
    x0 += 8 * C::kLd;
  }
}

template <typename T, int DP>
__device__ __forceinline__ void store_acc_row(T* dst, const float4 (&acc)[Tiled<DP>::kND], float scale, int d, int tx) {
#pragma unroll
  for (int j = 0; j < Tiled<DP>::kND; ++j) {
    const int c = tx * 4 + 64 * j;
    if (c + 0 < d) dst[c + 0] = from_f32<T>(acc[j].x * scale);
    if (c + 1 < d) dst[c + 1] = from_f32<T>(acc[j].y * scale);
    if (c + 2 < d) dst[c + 2] = from_f32<T>(acc[j].z * scale);
    if (c + 3 < d) dst[c + 3] = from_f32<T>(acc[j].w * scale);
  }
}

// Keep bits of a thread's scores when rows are queries: the four lanes of a quad own the four keys of
// a Philox counter for each (row, j); each lane draws one of the quad's four rows and they exchange.
// Bit 4*j + i of the result: row ty*4 + i, column tx + 16 j.
template <int NC>
__device__ __forceinline__ uint32_t tile_keep_bits(const DropoutCtx& d, int m_first, int n_first, int tx) {
  const int lane = threadIdx.x & 31, q = lane & 3;
  uint32_t mine = 0u, keep = 0u;
#pragma unroll
  for (int j = 0; j < NC; ++j) mine |= dropout_keep4(d, m_first + q, (n_first + (tx & ~3) + 16 * j) >> 2) << (4 * j);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = __shfl_sync(0xffffffffu, mine, (lane & ~3) | i);
#pragma unroll
    for (int j = 0; j < NC; ++j) keep |= ((w >> (4 * j + q)) & 1u) << (4 * j + i);
  }
  return keep;
}

template <typename T>
__device__ __forceinline__ const T* bias_at(const Params& p, const Seq& sq, int h, int m, int n) {
  return reinterpret_cast<const T*>(p.bias.ptr) + (int64_t)sq.bidx * p.bias.s[0] + (int64_t)h * p.bias.s[1] +
         (int64_t)m * p.bias.s[2] + (int64_t)n * p.bias.s[3];
}

// Forward.  grid = (cdiv(max_sq, 32), Hq, batch).  Two groups of four warps take every other block of the keys, each with
// tiles of its own, and merge at the end: a row tile's chain of blocks, which is what a small grid waits for, is half
// as long, and an SM has 16 warps instead of 12.  Within a group the copy of V runs under the scores, that of the next K
// under the accumulation.
constexpr int kFwdGroups = 2;
template <typename T, int DP>
__global__ void __launch_bounds__(kFwdGroups * 128, 2) tiled_fwd_kernel(const __grid_constant__ Params p) {
  wait_for_earlier_grids();
  using C = Tiled<DP>;
  constexpr int kGroupFloats = 2 * C::kBN * C::kLd + C::kBM * C::kLdP;
  extern __shared__ float smem[];
  const int grp = threadIdx.x >> 7, tid = threadIdx.x & 127;
  float* Qs = smem;                                              // [32][LD]
  float* Ks = Qs + C::kBM * C::kLd + grp * kGroupFloats;         // [BN][LD]
  float* Vs = Ks + C::kBN * C::kLd;                              // [BN][LD]
  float* Ps = Vs + C::kBN * C::kLd;                              // [32][BN + 4]
  // One thread of the grid reports the seed and offset actually used, before any early exit
  // (the first sequence of a varlen batch may be empty).
  if (p.dropout_on && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0) {
    if (p.seed_out) *p.seed_out = p.seed_ptr ? *p.seed_ptr : 0ull;
    if (p.off_out) *p.off_out = p.off2 + (p.off1_ptr ? *p.off1_ptr : 0ull);
  }
  int x, h, z;
  tile_of_block<true>((int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, (int)gridDim.x, (int)gridDim.y, (int)gridDim.z, x, h, z);
  const int m0 = ((int)gridDim.x - 1 - x) * C::kBM;
  const Seq sq = resolve_seq(p, z);
  if (m0 >= sq.sq) return;
  const int hk = h / p.group, ty = tid >> 4, tx = tid & 15;
  const bool kvec = rows_vec4<T>(p.k, p.dqk), vvec = rows_vec4<T>(p.v, p.dvo);
  auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); };
  DropoutCtx dctx;
  if (p.dropout_on) dctx = dropout_ctx(p, z, h);
  int n_lo, n_hi, w_lo = 1, w_hi = 0;
  key_range(p, sq, m0, min(m0 + C::kBM, sq.sq) - 1, n_lo, n_hi);
  const int wm = m0 + (tid >> 5) * kWarpRows;
  if (wm < sq.sq) key_range(p, sq, wm, min(wm + kWarpRows, sq.sq) - 1, w_lo, w_hi);
  const int d4 = (p.dqk + 3) >> 2;
  int n0 = n_lo / C::kBN * C::kBN + grp * C::kBN;
  stage_tile<T, DP, C::kBM, kFwdGroups * 128>(Qs, p.q, sq.bidx, h, sq.q0, m0, sq.sq, p.dqk, rows_vec4<T>(p.q, p.dqk), threadIdx.x);
  if (n0 <= n_hi) stage_tile<T, DP, C::kBN, 128>(Ks, p.k, sq.bidx, hk, sq.k0, n0, sq.sk, p.dqk, kvec, tid);
  float m_i[4], l_i[4];
  float4 acc[4][C::kND];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_i[i] = -INFINITY;
    l_i[i] = 0.f;
#pragma unroll
    for (int j = 0; j < C::kND; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  stage_wait<0>();
  __syncthreads();      // (Q is staged by both groups)
  for (; n0 <= n_hi; n0 += kFwdGroups * C::kBN) {
    stage_wait<0>();
    group_sync();       // K has landed, the previous block's V has been read
    stage_tile<T, DP, C::kBN, 128>(Vs, p.v, sq.bidx, hk, sq.k0, n0, sq.sk, p.dvo, vvec, tid);
    float s[4][C::kNC];
    tile_dots<DP>(s, Qs, Ks, d4, ty, tx);
    const uint32_t keep = p.dropout_on ? tile_keep_bits<C::kNC>(dctx, m0 + ty * 4, n0, tx) : 0xffffffffu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + ty * 4 + i;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < C::kNC; ++j) {
        const int n = n0 + tx + 16 * j;
        const bool ok = score_valid(p, sq, m, n);
        s[i][j] *= p.qk_scale;
        if (ok && p.has_bias) s[i][j] += to_f32<T>(*bias_at<T>(p, sq, h, m, n)) * kLog2e;
        if (!ok) s[i][j] = -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
      const float m_new = fmaxf(m_i[i], half_warp_max(mx));
      const float ms = m_new == -INFINITY ? 0.f : m_new, alpha = exp2f(m_i[i] - ms);   // m_i == -inf -> 0
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < C::kNC; ++j) {
        float pv = exp2f(s[i][j] - ms);
        sum += pv;
        if (!((keep >> (4 * j + i)) & 1u)) pv = 0.f;
        Ps[(ty * 4 + i) * C::kLdP + tx + 16 * j] = round_to<T>(pv);
      }
      l_i[i] = l_i[i] * alpha + sum;      // this lane's columns: the row's sums meet after the loop
      m_i[i] = m_new;
#pragma unroll
      for (int j = 0; j < C::kND; ++j) {
        acc[i][j].x *= alpha; acc[i][j].y *= alpha; acc[i][j].z *= alpha; acc[i][j].w *= alpha;
      }
    }
    stage_wait<0>();
    group_sync();       // V has landed, K has been read
    if (n0 + kFwdGroups * C::kBN <= n_hi)
      stage_tile<T, DP, C::kBN, 128>(Ks, p.k, sq.bidx, hk, sq.k0, n0 + kFwdGroups * C::kBN, sq.sk, p.dqk, kvec, tid);
    int k0, k1;
    seen_columns<DP>(w_lo, w_hi, n0, k0, k1);
    tile_accumulate<DP>(acc, Ps, Vs, k0, k1, ty, tx);
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) l_i[i] = half_warp_sum(l_i[i]);
  // The second group's sums reach the first through the second's own K tile (every warp of the group has read the last
  // one), a row's maximum and sum in the padding behind it.
  float* theirs = Qs + C::kBM * C::kLd + kGroupFloats;
  if (grp == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty * 4 + i;
#pragma unroll
      for (int j = 0; j < C::kND; ++j) *reinterpret_cast<float4*>(theirs + r * C::kLd + tx * 4 + 64 * j) = acc[i][j];
      if (tx == 0) *reinterpret_cast<float2*>(theirs + r * C::kLd + DP) = make_float2(m_i[i], l_i[i]);
    }
  }
  __syncthreads();
  if (grp == 1) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i, m = m0 + r;
    const float2 o = *reinterpret_cast<const float2*>(theirs + r * C::kLd + DP);
    const float mx = fmaxf(m_i[i], o.x), ms = mx == -INFINITY ? 0.f : mx;
    const float mine = exp2f(m_i[i] - ms), other = exp2f(o.x - ms);      // (-inf: no key in that half -> 0)
    const float l = l_i[i] * mine + o.y * other;
    if (m >= sq.sq) continue;
#pragma unroll
    for (int j = 0; j < C::kND; ++j) {
      const float4 t = *reinterpret_cast<const float4*>(theirs + r * C::kLd + tx * 4 + 64 * j);
      acc[i][j].x = acc[i][j].x * mine + t.x * other;
      acc[i][j].y = acc[i][j].y * mine + t.y * other;
      acc[i][j].z = acc[i][j].z * mine + t.z * other;
      acc[i][j].w = acc[i][j].w * mine + t.w * other;
    }
    // natural-log LSE of the scaled, biased logits; rows without any valid key get O = 0, LSE = +inf
    if (tx == 0 && p.lse != nullptr) p.lse[lse_offset(p, sq, h) + m] = l > 0.f ? (mx + log2f(l)) * kLn2 : INFINITY;
    store_acc_row<T, DP>(row_ptr_mut<T>(p.out, sq.bidx, h, sq.q0 + m), acc[i], l > 0.f ? (1.f / l) * p.dropout_scale : 0.f, p.dvo, tx);
  }
}

// SPLIT 2: two CTAs of a cluster take every other block of the other sequence dimension and exchange their sums at the end, each
// finishing one half of the result.  A row tile's chain of blocks is then half as long: where the grid does not fill the
// chip several times over, the longest chain is the launch's time (split_backward()).
__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// This thread's N float4 of `give` go to the same thread of the other CTA, whose are added to `keep`.  `buf`: 128 * N float4 that nobody
// reads or copies to any more.
template <int N>
__device__ __forceinline__ void pair_exchange(float* buf, float4 (&keep)[N], const float4 (&give)[N], uint32_t rank) {
#pragma unroll
  for (int n = 0; n < N; ++n) *reinterpret_cast<float4*>(buf + 4 * (n * 128 + (int)threadIdx.x)) = give[n];
  pair_sync();
  const uint32_t addr = ptx::smem_u32(buf + 4 * threadIdx.x);
#pragma unroll
  for (int n = 0; n < N; ++n) {
    float4 v;
    asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [a];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr + 2048 * n), "r"(rank ^ 1u) : "memory");
    keep[n].x += v.x; keep[n].y += v.y; keep[n].z += v.z; keep[n].w += v.w;
  }
  pair_sync();      // (the other CTA may still be reading)
}

// dK / dV of 32 keys of one kv head.  The scores of dO V^T come first: its tile is the first to be free again, so that the
// next block's dO is on its way under the accumulation of dK, Q behind it.
template <typename T, int DP, int SPLIT>
__device__ __forceinline__ void tiled_bwd_dkdv(const Params& p, float* smem, int z, int hk, int n0) {
  using C = Tiled<DP>;
  constexpr int kThr = C::kThreads;
  float* Ks = smem;                       // [32][LD]
  float* Vs = Ks + C::kBM * C::kLd;
  float* Qs = Vs + C::kBM * C::kLd;       // [BN][LD]
  float* dOs = Qs + C::kBN * C::kLd;
  float* Ps = dOs + C::kBN * C::kLd;      // [32][BN + 4]
  float* dSs = Ps + C::kBM * C::kLdP;
  float* lse_s = dSs + C::kBM * C::kLdP;  // [BN]
  float* dl_s = lse_s + C::kBN;
  const Seq sq = resolve_seq(p, z);
  if (n0 >= sq.sk) return;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const bool qvec = rows_vec4<T>(p.q, p.dqk), dovec = rows_vec4<T>(p.dout, p.dvo);
  float4 adv[4][C::kND], adk[4][C::kND];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < C::kND; ++j) adv[i][j] = adk[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
  int m_lo, m_hi, w_lo = 1, w_hi = 0;
  query_range(p, sq, n0, min(n0 + C::kBM, sq.sk) - 1, m_lo, m_hi);
  const int wn = n0 + (tid >> 5) * kWarpRows;
  if (wn < sq.sk) query_range(p, sq, wn, min(wn + kWarpRows, sq.sk) - 1, w_lo, w_hi);
  const int dq4 = (p.dqk + 3) >> 2, dv4 = (p.dvo + 3) >> 2;
  const int first = m_lo / C::kBN * C::kBN;
  auto stage_q = [&](int h, int m0) {      // Q, and the rows' logsumexp and delta
    stage_tile<T, DP, C::kBN, kThr>(Qs, p.q, sq.bidx, h, sq.q0, m0, sq.sq, p.dqk, qvec, tid);
    if (tid < C::kBN) {
      const int m = m0 + tid;
      const int64_t lrow = lse_offset(p, sq, h);
      lse_s[tid] = m < sq.sq ? p.lse[lrow + m] * kLog2e : INFINITY;
      dl_s[tid] = m < sq.sq ? p.delta[lrow + m] : 0.f;
    }
  };
  auto stage_do = [&](int h, int m0) {
    stage_tile<T, DP, C::kBN, kThr>(dOs, p.dout, sq.bidx, h, sq.q0, m0, sq.sq, p.dvo, dovec, tid);
  };
  const uint32_t rank = SPLIT == 2 ? pair_rank() : 0u;
  const int nblk = m_lo <= m_hi ? m_hi / C::kBN - m_lo / C::kBN + 1 : 0, total = nblk * p.group;
  int g = 0, mb = 0;      // head of the group and block of it
  auto advance = [&] { if (++mb == nblk) { mb = 0; ++g; } };
  if (rank == 1) advance();
  if ((int)rank < total) {
    stage_tile<T, DP, C::kBM, kThr>(Vs, p.v, sq.bidx, hk, sq.k0, n0, sq.sk, p.dvo, rows_vec4<T>(p.v, p.dvo), tid);
    stage_do(hk * p.group + g, first + mb * C::kBN);
    stage_tile<T, DP, C::kBM, kThr>(Ks, p.k, sq.bidx, hk, sq.k0, n0, sq.sk, p.dqk, rows_vec4<T>(p.k, p.dqk), tid);
    stage_wait<1>();      // V and dO
    __syncthreads();
    stage_q(hk * p.group + g, first + mb * C::kBN);
  }
  for (int i = (int)rank; i < total; i += SPLIT) {
    {
      const int h = hk * p.group + g, m0 = first + mb * C::kBN;
      DropoutCtx dctx;
      if (p.dropout_on) dctx = dropout_ctx(p, z, h);
#pragma unroll
      for (int u = 0; u < SPLIT; ++u) advance();
      const bool more = i + SPLIT < total;
      const int next_h = hk * p.group + g, next_m0 = first + mb * C::kBN;
      float s[4][C::kNC], dp[4][C::kNC];
      tile_dots<DP>(dp, Vs, dOs, dv4, ty, tx);
      stage_wait<0>();
      __syncthreads();      // K, Q, logsumexp and delta are there
      tile_dots<DP>(s, Ks, Qs, dq4, ty, tx);
#pragma unroll
      for (int j = 0; j < C::kNC; ++j) {
        const int c = tx + 16 * j, m = m0 + c;
        // (a thread's four keys are the four columns of one Philox counter)
        const uint32_t keep = p.dropout_on ? dropout_keep4(dctx, m, (n0 + ty * 4) >> 2) : 15u;
        const float lse = lse_s[c], dl = dl_s[c];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = n0 + ty * 4 + i;
          float pd = 0.f, ds = 0.f;
          if (score_valid(p, sq, m, n)) {
            float x = s[i][j] * p.qk_scale;
            if (p.has_bias) x += to_f32<T>(*bias_at<T>(p, sq, h, m, n)) * kLog2e;
            const float pr = exp2f(x - lse);      // lse = +inf on dead rows -> 0
            const bool kept = (keep >> i) & 1u;
            pd = kept ? pr * p.dropout_scale : 0.f;
            ds = pr * ((kept ? dp[i][j] * p.dropout_scale : 0.f) - dl);
          }
          Ps[(ty * 4 + i) * C::kLdP + c] = round_to<T>(pd);
          dSs[(ty * 4 + i) * C::kLdP + c] = round_to<T>(ds);
        }
      }
      __syncwarp();
      int k0, k1;
      seen_columns<DP>(w_lo, w_hi, m0, k0, k1);
      tile_accumulate<DP>(adv, Ps, dOs, k0, k1, ty, tx);
      __syncthreads();      // dO has been read
      if (more) stage_do(next_h, next_m0);
      tile_accumulate<DP>(adk, dSs, Qs, k0, k1, ty, tx);
      stage_wait<0>();
      __syncthreads();      // Q has been read, the next dO is there
      if (more) stage_q(next_h, next_m0);
    }
  }
  if constexpr (SPLIT == 2) {      // the first CTA finishes dK, the second dV (Q's and dO's tiles are free)
    float4 mine[4 * C::kND], theirs[4 * C::kND];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < C::kND; ++j) {
        mine[i * C::kND + j] = rank == 0 ? adk[i][j] : adv[i][j];
        theirs[i * C::kND + j] = rank == 0 ? adv[i][j] : adk[i][j];
      }
    pair_exchange<4 * C::kND>(Qs, mine, theirs, rank);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = n0 + ty * 4 + i;
      if (n >= sq.sk) continue;
      float4 row[C::kND];
#pragma unroll
      for (int j = 0; j < C::kND; ++j) row[j] = mine[i * C::kND + j];
      store_acc_row<T, DP>(row_ptr_mut<T>(rank == 0 ? p.dk : p.dv, sq.bidx, hk, sq.k0 + n), row, rank == 0 ? p.sm_scale : 1.f, rank == 0 ? p.dqk : p.dvo, tx);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = n0 + ty * 4 + i;
    if (n >= sq.sk) continue;
    store_acc_row<T, DP>(row_ptr_mut<T>(p.dk, sq.bidx, hk, sq.k0 + n), adk[i], p.sm_scale, p.dqk, tx);
    store_acc_row<T, DP>(row_ptr_mut<T>(p.dv, sq.bidx, hk, sq.k0 + n), adv[i], 1.f, p.dvo, tx);
  }
}

// dQ (+ dBias) of 32 query rows of one head.  V is read by the scores only: the next block's is on its way for the rest
// of a block.
template <typename T, int DP, int SPLIT>
__device__ __forceinline__ void tiled_bwd_dq(const Params& p, float* smem, int z, int h, int m0) {
  using C = Tiled<DP>;
  constexpr int kThr = C::kThreads;
  float* Qs = smem;                       // [32][LD]
  float* dOs = Qs + C::kBM * C::kLd;
  float* Ks = dOs + C::kBM * C::kLd;      // [BN][LD]
  float* Vs = Ks + C::kBN * C::kLd;
  float* dSs = Vs + C::kBN * C::kLd;      // [32][BN + 4]
  const Seq sq = resolve_seq(p, z);
  if (m0 >= sq.sq) return;
  const int tid = threadIdx.x, hk = h / p.group, ty = tid >> 4, tx = tid & 15;
  const bool kvec = rows_vec4<T>(p.k, p.dqk), vvec = rows_vec4<T>(p.v, p.dvo);
  DropoutCtx dctx;
  if (p.dropout_on) dctx = dropout_ctx(p, z, h);
  int n_lo, n_hi, w_lo = 1, w_hi = 0;
  key_range(p, sq, m0, min(m0 + C::kBM, sq.sq) - 1, n_lo, n_hi);
  const uint32_t rank = SPLIT == 2 ? pair_rank() : 0u;
  const int first = n_lo / C::kBN * C::kBN + (int)rank * C::kBN;      // (this CTA's)
  auto stage_k = [&](int n0) { stage_tile<T, DP, C::kBN, kThr>(Ks, p.k, sq.bidx, hk, sq.k0, n0, sq.sk, p.dqk, kvec, tid); };
  auto stage_v = [&](int n0) { stage_tile<T, DP, C::kBN, kThr>(Vs, p.v, sq.bidx, hk, sq.k0, n0, sq.sk, p.dvo, vvec, tid); };
  if (first <= n_hi) {
    stage_tile<T, DP, C::kBM, kThr>(dOs, p.dout, sq.bidx, h, sq.q0, m0, sq.sq, p.dvo, rows_vec4<T>(p.dout, p.dvo), tid);
    stage_v(first);
    stage_tile<T, DP, C::kBM, kThr>(Qs, p.q, sq.bidx, h, sq.q0, m0, sq.sq, p.dqk, rows_vec4<T>(p.q, p.dqk), tid);
    stage_k(first);
  }
  const int64_t lrow = lse_offset(p, sq, h);
  float lse[4], dl[4];
  float4 adq[4][C::kND];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    lse[i] = m < sq.sq ? p.lse[lrow + m] * kLog2e : INFINITY;
    dl[i] = m < sq.sq ? p.delta[lrow + m] : 0.f;
#pragma unroll
    for (int j = 0; j < C::kND; ++j) adq[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int wm = m0 + (tid >> 5) * kWarpRows;
  if (wm < sq.sq) key_range(p, sq, wm, min(wm + kWarpRows, sq.sq) - 1, w_lo, w_hi);
  if (rank == 0) {
    if (n_hi >= n_lo) zero_dbias_outside<T>(p, sq, h, m0, C::kBM, n_lo / C::kBN * C::kBN, (n_hi / C::kBN + 1) * C::kBN);
    else zero_dbias_outside<T>(p, sq, h, m0, C::kBM, 0, 0);
  }
  const int dq4 = (p.dqk + 3) >> 2, dv4 = (p.dvo + 3) >> 2;
  stage_wait<2>();      // dO and V
  __syncthreads();
  for (int n0 = first; n0 <= n_hi; n0 += SPLIT * C::kBN) {
    const bool more = n0 + SPLIT * C::kBN <= n_hi;
    float s[4][C::kNC], dp[4][C::kNC];
    tile_dots<DP>(dp, dOs, Vs, dv4, ty, tx);
    stage_wait<0>();
    __syncthreads();      // V has been read, K (and Q) is there
    if (more) stage_v(n0 + SPLIT * C::kBN);
    tile_dots<DP>(s, Qs, Ks, dq4, ty, tx);
    const uint32_t keep = p.dropout_on ? tile_keep_bits<C::kNC>(dctx, m0 + ty * 4, n0, tx) : 0xffffffffu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + ty * 4 + i;
#pragma unroll
      for (int j = 0; j < C::kNC; ++j) {
        const int n = n0 + tx + 16 * j;
        float ds = 0.f;
        if (score_valid(p, sq, m, n)) {
          float x = s[i][j] * p.qk_scale;
          if (p.has_bias) x += to_f32<T>(*bias_at<T>(p, sq, h, m, n)) * kLog2e;
          const float pr = exp2f(x - lse[i]);
          ds = pr * (((keep >> (4 * j + i)) & 1u ? dp[i][j] * p.dropout_scale : 0.f) - dl[i]);
        }
        if (p.has_dbias && m < sq.sq && n < sq.sk) {
          T* dbp = reinterpret_cast<T*>(p.dbias.ptr) + (int64_t)sq.bidx * p.dbias.s[0] + (int64_t)h * p.dbias.s[1] +
                   (int64_t)m * p.dbias.s[2] + (int64_t)n * p.dbias.s[3];
          *dbp = from_f32<T>(ds);
        }
        dSs[(ty * 4 + i) * C::kLdP + tx + 16 * j] = round_to<T>(ds);
      }
    }
    __syncwarp();
    int k0, k1;
    seen_columns<DP>(w_lo, w_hi, n0, k0, k1);
    tile_accumulate<DP>(adq, dSs, Ks, k0, k1, ty, tx);
    stage_wait<0>();
    __syncthreads();      // K has been read, the next V is there
    if (more) stage_k(n0 + SPLIT * C::kBN);
  }
  if constexpr (SPLIT == 2) {      // the first CTA finishes two of a thread's rows, the second the others (K's and V's tiles are free)
    float4 mine[2 * C::kND], theirs[2 * C::kND];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < C::kND; ++j) {
        mine[i * C::kND + j] = rank == 0 ? adq[i][j] : adq[i + 2][j];
        theirs[i * C::kND + j] = rank == 0 ? adq[i + 2][j] : adq[i][j];
      }
    pair_exchange<2 * C::kND>(Ks, mine, theirs, rank);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int m = m0 + ty * 4 + 2 * (int)rank + i;
      float4 row[C::kND];
#pragma unroll
      for (int j = 0; j < C::kND; ++j) row[j] = mine[i * C::kND + j];
      if (m < sq.sq) store_acc_row<T, DP>(row_ptr_mut<T>(p.dq, sq.bidx, h, sq.q0 + m), row, p.sm_scale, p.dqk, tx);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m < sq.sq) store_acc_row<T, DP>(row_ptr_mut<T>(p.dq, sq.bidx, h, sq.q0 + m), adq[i], p.sm_scale, p.dqk, tx);
  }
}

// The backward.  WHICH 1: dK / dV, grid = (cdiv(max_sk, 32), Hk, batch).  2: dQ (+ dBias), grid = (cdiv(max_sq, 32),
// Hq, batch), last rows first.  3: both in one launch, x alternating between the two (neither reads what the other
// writes); joint_backward() says when.  At the sizes single precision is used at, each of the two alone leaves most of the chip idle: 2 x 8
// heads x 500 tokens are 256 CTAs of four warps, 7 warps an SM, waiting for their own loads and barriers.
template <typename T, int DP, int WHICH, int SPLIT>
__global__ void __cluster_dims__(SPLIT, 1, 1) __launch_bounds__(128, DP <= 64 || WHICH == 2 ? 3 : 2)
tiled_bwd_kernel(const __grid_constant__ Params p) {
  wait_for_earlier_grids();
  extern __shared__ float smem[];
  constexpr int kBM = Tiled<DP>::kBM;
  const int nx = (int)gridDim.x / SPLIT;
  int x, h, z;
  tile_of_block<false>((int)blockIdx.x / SPLIT, (int)blockIdx.y, (int)blockIdx.z, nx, (int)gridDim.y, (int)gridDim.z, x, h, z);
  if constexpr (WHICH == 1) {
    tiled_bwd_dkdv<T, DP, SPLIT>(p, smem, z, h, x * kBM);
  } else if constexpr (WHICH == 2) {
    tiled_bwd_dq<T, DP, SPLIT>(p, smem, z, h, (nx - 1 - x) * kBM);
  } else {
    if (x & 1) {
      const int m0 = (nx / 2 - 1 - (x >> 1)) * kBM;
      if (m0 < p.max_sq) tiled_bwd_dq<T, DP, SPLIT>(p, smem, z, h, m0);
    } else if (h < p.hk) {
      tiled_bwd_dkdv<T, DP, SPLIT>(p, smem, z, h, (x >> 1) * kBM);
    }
  }
}
