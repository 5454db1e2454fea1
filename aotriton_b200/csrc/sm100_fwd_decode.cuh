// Forward attention for a handful of query rows against a long key/value sequence (decoding, chunks of
// a few tokens).  Included by sm100_fwd.cu inside its namespaces.
//
// What bounds it: reading K and V once.  The tile kernel gives each (sequence, q head) one CTA, whose
// 128-row tile then holds one or a few rows: a sequence's keys are walked by group_size CTAs one after
// another, each K/V block waiting for the chain of two GEMMs and a softmax behind it, and a batch of a
// few sequences leaves most of the chip idle (4 sequences x 6007 keys, 32:8 heads of 128, bf16: 133 us,
// 0.74 TB/s).  Here
//   * the query heads of one kv head are packed into the rows of one tile (row r = head r / sq of the
//     group, query r % sq), so that K and V are read once per kv head and not once per q head;
//   * the keys of one (sequence, kv head) are cut into CS contiguous pieces, one CTA of a cluster each
//     (CS up to 8); the pieces' partial results (row maximum, row sum, unnormalised O) meet in
//     distributed shared memory, so the split needs no workspace and no second launch;
//   * a CTA streams its piece in tiles of 64 keys through a ring of TMA copies, deep enough to keep the
//     memory busy (two CTAs per SM: about 190 KB on the way); four warps take 16 keys of a tile each and
//     keep a running softmax of their own, so nothing inside the stream waits for another warp.
// The products are 16 rows high, where the 128-row tensor-memory MMA would compute padding and add its
// read-out latency to every tile: they run as warp-level m16n8k16 MMAs from registers and ldmatrix.
//
// Every wait inside a CTA is bounded.  A CTA whose wait ran out, or that starts after a failure, still takes both
// cluster barriers, so its peers do not wait for it.
//
// Arithmetic as in the tile kernel: scores scaled by sm_scale*log2(e) in fp32, masked scores -inf, P cast to
// the value type before P V, fp32 sums, rows without a key give O = 0, LSE = +inf.

constexpr int kDecodeMaxQueries = 16;   // the longest query sequence that comes here
constexpr int kDecKeys = 64;             // keys per tile: 16 for each consumer warp

// W consumer warps (four per tile: with eight, warps 4-7 take the odd tiles) and one TMA producer.
template <int HD, int MT, int W>
struct DecSmem {
  static constexpr int kThreads = (W + 1) * 32;
  static constexpr int kRows = 16 * MT;                      // query rows of a CTA
  static constexpr int kCtasPerSm = W > 4 || (HD > 64 && MT > 1) ? 1 : 2;   // (32 rows x 128 columns of O and Q take 200 registers)
  static constexpr int kTile = (HD / 64) * kDecKeys * 128;   // 64 keys x HD x 2 bytes, 64-column boxes
  static constexpr int kMaxStages = HD > 64 ? 6 : 12;        // 192 KB of K and V on the way; half of it with two CTAs per SM
  static constexpr int bFull = 0, bEmpty = kMaxStages, bCount = 2 * kMaxStages;
  static constexpr int kBars = 0;
  static constexpr int kAbort = kBars + bCount * 8;
  static constexpr int kMl = (kAbort + 8 + 15) & ~15;        // per warp: row maxima and sums; the CTA's after the merge
  static constexpr int kMlFloats = (W + 1) * 2 * kRows;
  static constexpr int kRing = (kMl + kMlFloats * 4 + 1023) & ~1023;   // stages: K tile, V tile
  static constexpr int dynamic(int stages) { return kRing + stages * 2 * kTile + 1024; }
  // The ring is idle once the stream has ended: the partial O of each warp goes there (rows padded by
  // four floats against bank conflicts), the CTA's merged O behind them.
  static constexpr int kLdO = HD + 4;
  static constexpr int kOWarp = kRows * kLdO;                // floats per partial
  static_assert((W + 1) * kOWarp * 4 <= kMaxStages / kCtasPerSm * 2 * kTile, "partials fit in the ring");
};

template <typename T>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t saddr, uint32_t rank) {
  float v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
               : "=f"(v) : "r"(saddr), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t saddr, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(saddr), "r"(rank) : "memory");
  return v;
}

// grid = (CS, Hk * row chunks, batch); cluster = the CS CTAs of one x row
template <typename T, int HD, int MT, int CS, int W>
__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(DecSmem<HD, MT, W>::kThreads, DecSmem<HD, MT, W>::kCtasPerSm)
sm100_fwd_decode_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_v, unsigned int* status, int stages) {
  wait_for_earlier_grids();
  using L = DecSmem<HD, MT, W>;
  constexpr int kBoxes = HD / 64, kKsteps = HD / 16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kAbort);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.z;
  const int hk = (int)blockIdx.y % p.hk, chunk = (int)blockIdx.y / p.hk;
  const uint32_t rank = CS > 1 ? cluster_rank() : 0u;
  // Everything up to the stream depends on the sequence, the head and the chunk only: a cluster leaves
  // here as a whole or not at all.
  const Seq sq = resolve_seq(p, z);
  const int rows_total = p.group * sq.sq, row0 = chunk * L::kRows;
  if (row0 >= rows_total) return;
  const int nrows = min(L::kRows, rows_total - row0);
  // queries of the chunk's rows: [m_lo, m_hi] (the whole range as soon as the rows span two heads)
  int m_lo = row0 % sq.sq, m_hi = (row0 + nrows - 1) % sq.sq;
  if (row0 / sq.sq != (row0 + nrows - 1) / sq.sq) { m_lo = 0; m_hi = sq.sq - 1; }
  int n_lo, n_hi;
  key_range(p, sq, m_lo, m_hi, n_lo, n_hi);
  const int t_lo = n_lo / kDecKeys;
  const int ntiles = n_hi < n_lo ? 0 : n_hi / kDecKeys - t_lo + 1;
  // this CTA's share of the tiles
  const int first = (int)((int64_t)ntiles * rank / CS), last = (int)((int64_t)ntiles * (rank + 1) / CS);

  if (threadIdx.x == 0) {
    init_abort_and_limit(abort_flag, p.wait_limit_kcycles);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&bars[L::bFull + s], 1);
      mbar_init(&bars[L::bEmpty + s], 4);
    }
    fence_barrier_init();
  }
  // After an earlier failure the CTA streams nothing, but it takes both cluster barriers: a peer may read
  // its shared memory.
  const bool dead = __syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile unsigned int*>(status) != 0u);
  const int n = dead ? 0 : last - first;

  float* ml = reinterpret_cast<float*>(smem + L::kMl);
  float* po = reinterpret_cast<float*>(smem + L::kRing);
  if (warp == W) {
    // ================================ TMA producer ===================================
    if (lane == 0) {
      int issued = 0;
      for (int i = 0, s = 0, ph = 1; i < n; ++i) {      // s, ph: ring stage and the parity that frees it
        const int krow = (int)(sq.k0 + (int64_t)(t_lo + first + i) * kDecKeys);
        if (!mbar_wait(&bars[L::bEmpty + s], (uint32_t)ph, abort_flag, status, 0x5000)) break;
        if (!(p.drop_copy == 1 && i == 0 && rank == 0)) {      // (test hook: the cluster's first tile never arrives)
          uint8_t* kt = smem + L::kRing + s * (2 * L::kTile);
          mbar_expect_tx(&bars[L::bFull + s], 2 * L::kTile);
          for (int b = 0; b < kBoxes; ++b)
            tma_load_4d(kt + b * (kDecKeys * 128), &tm_k, &bars[L::bFull + s], b * 64, krow, hk, sq.bidx);
          for (int b = 0; b < kBoxes; ++b)
            tma_load_4d(kt + L::kTile + b * (kDecKeys * 128), &tm_v, &bars[L::bFull + s], b * 64, krow, hk, sq.bidx);
          issued = i + 1;
        }
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      if (*abort_flag) {      // let copies that are still in flight land before the memory is used again
        for (int i = max(p.drop_copy == 1 && rank == 0 ? 1 : 0, issued - stages); i < issued; ++i)
          mbar_wait_quiet(&bars[L::bFull + i % stages], (uint32_t)(i / stages) & 1u, abort_flag);
      }
    }
    __syncwarp();
  }
  float m_run[2 * MT], l_run[2 * MT], o[MT][2 * kKsteps][4];
#pragma unroll
  for (int t = 0; t < MT; ++t) {
    m_run[2 * t] = m_run[2 * t + 1] = -INFINITY;
    l_run[2 * t] = l_run[2 * t + 1] = 0.f;
#pragma unroll
    for (int c = 0; c < 2 * kKsteps; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[t][c][e] = 0.f;
  }
  const int qr = lane >> 2, qc = (lane & 3) * 2;      // this lane's row (and row + 8) and column pair in a fragment
  if (warp < W && n > 0) {
    // ================================== consumer =====================================
    // Q as A fragments, straight from global memory (rows and columns beyond the ends are zero)
    uint32_t q[MT][kKsteps][4];
    int row_lo[2 * MT], row_hi[2 * MT];
#pragma unroll
    for (int t = 0; t < MT; ++t) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = t * 16 + half * 8 + qr;
        const bool in = r < nrows;
        const int rg = in ? row0 + r : row0;
        const int h = hk * p.group + rg / sq.sq, m = rg % sq.sq;
        const T* qp = reinterpret_cast<const T*>(p.q.ptr) + (int64_t)sq.bidx * p.q.s[0] + (int64_t)h * p.q.s[1] +
                      (sq.q0 + m) * p.q.s[2];
#pragma unroll
        for (int kk = 0; kk < kKsteps; ++kk)
#pragma unroll
          for (int c8 = 0; c8 < 2; ++c8) {
            const int d = kk * 16 + c8 * 8 + qc;
            q[t][kk][c8 * 2 + half] = (in && d < p.dqk) ? __ldg(reinterpret_cast<const uint32_t*>(qp + d)) : 0u;
          }
        int lo = 0, hi = sq.sk - 1;
        if (p.causal) {
          const int64_t l64 = (int64_t)m - sq.wl, h64 = (int64_t)m + sq.wr;
          if (l64 > lo) lo = (int)(l64 > 0x7fffffffLL ? 0x7fffffffLL : l64);
          if (h64 < hi) hi = (int)(h64 < -1 ? -1 : h64);
        }
        if (!in) { lo = 1; hi = 0; }
        row_lo[2 * t + half] = lo;
        row_hi[2 * t + half] = hi;
      }
    }
    const uint32_t smem_s = smem_u32(smem);
    // ldmatrix addresses inside a tile: 128-byte rows, 16-byte chunks XOR-swizzled with the row (the TMA
    // layout).  K: matrices (keys 0-7 | 8-15) x (d 0-7 | 8-15) of a 16 x 16 step; V, read transposed: the same.
    const int krow = (warp & 3) * 16 + (lane & 7) + ((lane >> 4) << 3), kchunk = (lane >> 3) & 1;
    const int vrow = (warp & 3) * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), vchunk = lane >> 4;
    for (int i = warp >> 2, s = warp >> 2, ph = 0; i < n; i += W / 4) {
      if (!__all_sync(0xffffffffu, mbar_wait(&bars[L::bFull + s], (uint32_t)ph, abort_flag, status, 0x5100))) break;
      const int key0 = (t_lo + first + i) * kDecKeys + (warp & 3) * 16;      // first key of this warp's 16
      const uint32_t kt = smem_s + L::kRing + s * (2 * L::kTile) + krow * 128;
      const uint32_t vt = smem_s + L::kRing + s * (2 * L::kTile) + L::kTile + vrow * 128;
      if (key0 + 16 > sq.sk) {
        // V rows beyond the sequence hold a neighbour's tokens or padding: a zero probability times a
        // non-finite value would poison the sum
        uint8_t* vtile = smem + L::kRing + s * (2 * L::kTile) + L::kTile;
        for (int rr = max(0, sq.sk - key0); rr < 16; ++rr)
          for (int c = lane; c < kBoxes * 8; c += 32)
            *reinterpret_cast<uint4*>(vtile + (c >> 3) * (kDecKeys * 128) + ((warp & 3) * 16 + rr) * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
        __syncwarp();
      }
      // (two accumulators per 8 keys with one tile of rows: half the chain of dependent MMAs)
      constexpr int kChains = MT == 1 ? 2 : 1;
      float sc[MT][2][4], sc2[2][4];
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[t][0][e] = sc[t][1][e] = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) sc2[0][e] = sc2[1][e] = 0.f;
#pragma unroll
      for (int kk = 0; kk < kKsteps; ++kk) {
        uint32_t kb[4];
        const int c = (kk & 3) * 2 + kchunk;
        ldsm4(kb, kt + (kk >> 2) * (kDecKeys * 128) + ((c ^ (krow & 7)) << 4));
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          const bool second = kChains == 2 && (kk & 1);
          mma_16816<T>(second ? sc2[0] : sc[t][0], q[t][kk], kb[0], kb[1]);
          mma_16816<T>(second ? sc2[1] : sc[t][1], q[t][kk], kb[2], kb[3]);
        }
      }
      if constexpr (kChains == 2) {
#pragma unroll
        for (int e = 0; e < 4; ++e) { sc[0][0][e] += sc2[0][e]; sc[0][1][e] += sc2[1][e]; }
      }
      uint32_t pa[MT][4];
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int nn = key0 + j * 8 + qc + (e & 1), half = e >> 1;
            const bool ok = nn >= row_lo[2 * t + half] && nn <= row_hi[2 * t + half];
            sc[t][j][e] = ok ? sc[t][j][e] * p.qk_scale : -INFINITY;
            mx[half] = fmaxf(mx[half], sc[t][j][e]);
          }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          mx[half] = fmaxf(mx[half], __shfl_xor_sync(0xffffffffu, mx[half], 1));
          mx[half] = fmaxf(mx[half], __shfl_xor_sync(0xffffffffu, mx[half], 2));
        }
        const bool grow = mx[0] > m_run[2 * t] || mx[1] > m_run[2 * t + 1];
        if (__any_sync(0xffffffffu, grow)) {
          float al[2];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const float mn = fmaxf(m_run[2 * t + half], mx[half]);
            al[half] = mn == -INFINITY ? 1.f : ex2(m_run[2 * t + half] - mn);
            m_run[2 * t + half] = mn;
            l_run[2 * t + half] *= al[half];
          }
#pragma unroll
          for (int c = 0; c < 2 * kKsteps; ++c) {
            o[t][c][0] *= al[0]; o[t][c][1] *= al[0];
            o[t][c][2] *= al[1]; o[t][c][3] *= al[1];
          }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const float ms = m_run[2 * t + half] == -INFINITY ? 0.f : m_run[2 * t + half];
          float sum = 0.f;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float e0 = ex2(sc[t][j][2 * half] - ms), e1 = ex2(sc[t][j][2 * half + 1] - ms);
            sum += e0 + e1;
            pa[t][2 * j + half] = pack2<T>(e0, e1);
          }
          l_run[2 * t + half] += sum;      // this lane's columns; the quad's sums meet after the stream
        }
      }
#pragma unroll
      for (int c = 0; c < kKsteps; ++c) {      // 16 columns of the head dim per step
        uint32_t vb[4];
        const int ch = (c & 3) * 2 + vchunk;
        ldsm4t(vb, vt + (c >> 2) * (kDecKeys * 128) + ((ch ^ (vrow & 7)) << 4));
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          mma_16816<T>(o[t][2 * c], pa[t], vb[0], vb[1]);
          mma_16816<T>(o[t][2 * c + 1], pa[t], vb[2], vb[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[L::bEmpty + s]);
      if ((s += W / 4) >= stages) { s -= stages; ph ^= 1; }      // (an even number of stages with eight warps)
    }
  }
  __syncthreads();      // the ring is idle: every tile has been read
  // ---- the CTA's partial: the four warps' results with a common row maximum ----------------------
  if (warp < W) {
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = t * 16 + half * 8 + qr;
        float l = l_run[2 * t + half];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if ((lane & 3) == 0) {
          ml[warp * 2 * L::kRows + r] = m_run[2 * t + half];
          ml[warp * 2 * L::kRows + L::kRows + r] = l;
        }
        float* dst = po + warp * L::kOWarp + r * L::kLdO + qc;
#pragma unroll
        for (int c = 0; c < 2 * kKsteps; ++c)
          *reinterpret_cast<float2*>(dst + c * 8) = make_float2(o[t][c][2 * half], o[t][c][2 * half + 1]);
      }
  }
  __syncthreads();
  float* mo = po + W * L::kOWarp;
  float* mml = ml + W * 2 * L::kRows;
  constexpr int kV4 = HD / 4;      // float4 columns of a row
  for (int i = threadIdx.x; i < nrows * kV4; i += L::kThreads) {
    const int r = i / kV4, c4 = (i - r * kV4) * 4;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < W; ++w) m = fmaxf(m, ml[w * 2 * L::kRows + r]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float a = m == -INFINITY ? 0.f : ex2(ml[w * 2 * L::kRows + r] - m);
      const float4 x = *reinterpret_cast<const float4*>(po + w * L::kOWarp + r * L::kLdO + c4);
      acc.x = fmaf(a, x.x, acc.x); acc.y = fmaf(a, x.y, acc.y);
      acc.z = fmaf(a, x.z, acc.z); acc.w = fmaf(a, x.w, acc.w);
      l = fmaf(a, ml[w * 2 * L::kRows + L::kRows + r], l);
    }
    *reinterpret_cast<float4*>(mo + r * L::kLdO + c4) = acc;
    if (c4 == 0) { mml[r] = m; mml[L::kRows + r] = l; }
  }
  // ---- the cluster's result: each CTA finishes its share of the rows' columns --------------------
  if constexpr (CS > 1) cluster_sync(); else __syncthreads();
  const uint32_t mo_s = smem_u32(mo), mml_s = smem_u32(mml);
  for (int i = (int)rank * L::kThreads + (int)threadIdx.x; i < nrows * kV4; i += CS * L::kThreads) {
    const int r = i / kV4, c4 = (i - r * kV4) * 4;
    float mk[CS], m = -INFINITY;
#pragma unroll
    for (int k = 0; k < CS; ++k) {
      mk[k] = CS > 1 ? ld_cluster_f32(mml_s + r * 4, k) : mml[r];
      m = fmaxf(m, mk[k]);
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
#pragma unroll
    for (int k = 0; k < CS; ++k) {
      const float a = m == -INFINITY ? 0.f : ex2(mk[k] - m);
      const float lk = CS > 1 ? ld_cluster_f32(mml_s + (L::kRows + r) * 4, k) : mml[L::kRows + r];
      const float4 x = CS > 1 ? ld_cluster_f32x4(mo_s + (r * L::kLdO + c4) * 4, k)
                              : *reinterpret_cast<const float4*>(mo + r * L::kLdO + c4);
      acc.x = fmaf(a, x.x, acc.x); acc.y = fmaf(a, x.y, acc.y);
      acc.z = fmaf(a, x.z, acc.z); acc.w = fmaf(a, x.w, acc.w);
      l = fmaf(a, lk, l);
    }
    const float inv = l > 0.f ? 1.f / l : 0.f;
    const int rg = row0 + r, h = hk * p.group + rg / sq.sq, mq = rg % sq.sq;
    if (!dead && c4 < p.dvo)
      *reinterpret_cast<uint2*>(reinterpret_cast<T*>(p.out.ptr) + (int64_t)sq.bidx * p.out.s[0] + (int64_t)h * p.out.s[1] +
                                (sq.q0 + mq) * p.out.s[2] + c4) =
          make_uint2(pack2<T>(acc.x * inv, acc.y * inv), pack2<T>(acc.z * inv, acc.w * inv));
    if (!dead && c4 == 0 && p.lse != nullptr)
      p.lse[lse_offset(p, sq, h) + mq] = l > 0.f ? (m + log2f(l)) * kLn2 : INFINITY;
  }
  if constexpr (CS > 1) cluster_sync();      // no CTA leaves while a peer may still read its partial
}

template <typename T, int HD, int MT, int CS, int W>
cudaError_t launch_decode_CS(const Params& p, int chunks, const CUtensorMap& tk, const CUtensorMap& tv, unsigned int* status,
                             int dev, bool remember, int stages, cudaStream_t st) {
  using L = DecSmem<HD, MT, W>;
  static std::atomic<bool> attr_set[64];
  if (!remember || !attr_set[dev].load(std::memory_order_acquire)) {
    cudaError_t e = host().func_set_smem(reinterpret_cast<const void*>(sm100_fwd_decode_kernel<T, HD, MT, CS, W>), L::dynamic(L::kMaxStages));
    if (e != cudaSuccess) return e;
    if (remember) attr_set[dev].store(true, std::memory_order_release);
  }
  cudaError_t e = launch_kernel(sm100_fwd_decode_kernel<T, HD, MT, CS, W>, dim3(CS, p.hk * chunks, p.batch), dim3(L::kThreads),
                                L::dynamic(stages), st, p, tk, tv, status, stages);
  if (e == cudaSuccess) count_launch();
  return e;
}

// How a call is cut: pieces of the keys (CTAs of a cluster), consumer warps of a CTA, ring stages, row chunks.
template <int HD, int MT>
SplitPlan split_plan(const Params& p, int sms) {
  using L = DecSmem<HD, MT, 4>;
  const int chunks = (p.group * p.max_sq + L::kRows - 1) / L::kRows;
  const int64_t clusters = (int64_t)p.hk * chunks * p.batch;
  const int tiles = (p.max_sk + kDecKeys - 1) / kDecKeys;
  // Cut the keys until the CTAs fill the chip once or a piece would fall below two tiles.  (More pieces than
  // that only add CTAs that wait for a slot: 2 x 8192 keys, 64:8 heads, 5 queries: 37 us with 4 pieces, 58 us with 8.)
  // The rule counts SMs; a cluster of eight also needs its SMs in one GPC, so a few counts just below the line leave
  // clusters for a second round (6007 keys, 8 heads of 128 per kv head: 15 clusters 12.4 us, 16 to 18 21 us, 19, with
  // four pieces, 16.5; 32 clusters 17.1, 34 to 37 30).
  int cs = 1;
  while (cs < 8 && clusters * cs * 2 <= (int64_t)L::kCtasPerSm * sms && tiles >= 4 * cs) cs *= 2;
  // With no more CTAs than SMs each gets the whole ring, and eight warps if its rows fit one tile: four warps
  // spend 1100 clocks on a tile of 64 keys, which is less than a CTA alone on its SM could be fed
  // (32768 keys, 32:8 heads of 128: 31 us with eight warps, 41 us with four).
  const bool alone = clusters * cs <= sms;
  return {cs, MT == 1 && alone && cs == 8 ? 8 : 4, alone ? L::kMaxStages : L::kMaxStages / L::kCtasPerSm, chunks};
}

template <typename T, int HD, int MT>
cudaError_t launch_decode_MT(const Params& p, cudaStream_t st) {
  CUtensorMap tk, tv;
  if (!make_tile_map_16bit(&tk, p.k, p.dqk, p.k.n[2], kDecKeys) || !make_tile_map_16bit(&tv, p.v, p.dvo, p.v.n[2], kDecKeys))
    return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  unsigned int* status = nullptr;
  bool remember = false;
  cudaError_t e = fwd_device_facts(&dev, &status, &sms, &remember);
  if (e != cudaSuccess) return e;
  const SplitPlan s = split_plan<HD, MT>(p, sms);
  if constexpr (MT == 1) {
    if (s.warps == 8) return launch_decode_CS<T, HD, 1, 8, 8>(p, s.chunks, tk, tv, status, dev, remember, s.stages, st);
  }
  switch (s.pieces) {
    case 1: return launch_decode_CS<T, HD, MT, 1, 4>(p, s.chunks, tk, tv, status, dev, remember, s.stages, st);
    case 2: return launch_decode_CS<T, HD, MT, 2, 4>(p, s.chunks, tk, tv, status, dev, remember, s.stages, st);
    case 4: return launch_decode_CS<T, HD, MT, 4, 4>(p, s.chunks, tk, tv, status, dev, remember, s.stages, st);
    default: return launch_decode_CS<T, HD, MT, 8, 4>(p, s.chunks, tk, tv, status, dev, remember, s.stages, st);
  }
}

inline bool decode_shape(const Params& p) {
  return p.max_sq <= kDecodeMaxQueries && p.dqk <= 128 && p.dvo <= 128 && !p.has_bias && !p.dropout_on;
}

// f<HD, MT>() of the instantiation that takes the call
template <typename F>
auto with_decode_tile(const Params& p, F f) {
  const bool small = p.dqk <= 64 && p.dvo <= 64, one = p.group * p.max_sq <= 16;
  if (small) return one ? f.template operator()<64, 1>() : f.template operator()<64, 2>();
  return one ? f.template operator()<128, 1>() : f.template operator()<128, 2>();
}

template <typename T>
cudaError_t launch_decode_T(const Params& p, cudaStream_t st) {
  return with_decode_tile(p, [&]<int HD, int MT>() { return launch_decode_MT<T, HD, MT>(p, st); });
}
