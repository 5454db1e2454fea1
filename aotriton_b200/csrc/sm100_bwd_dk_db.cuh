// dK of wide heads from a dBias that is already written: dK = sm_scale * dB^T Q.
// Included by sm100_bwd_wide.cuh inside its namespaces.
//
// Bias enters the scores with factor one, so dB is dS: the 16-bit values the dK kernel would form again (scores,
// exponentials, bias, keep bits, dP) to feed its accumulating GEMM.  When the caller wants dB, the dQ kernel runs
// before dK, and dK is left with one GEMM instead of three and with no compute warps at all.
//
// One CTA owns 128 keys of one kv head and walks the query rows that can see them, 64 at a time, over the q heads of
// the group.  Both operands are read the way they lie in memory, rows of queries: dB [64 x 128 keys] as the M-major
// A operand, Q [64 x head dim] as the N-major B operand.  A stage is 16 + 32 KB; two stages per CTA and two CTAs per
// SM (96 KB of shared memory, 256 columns of tensor memory each), so that one CTA's write-out and start run under the
// other's GEMMs.  Bounds: reading dB once (8 x 16 heads x 2048 x 2048: 1.07 GB, 0.17 ms) and the GEMM (0.16 ms).
// Measured, training step with bias and dropout 0.2, head dim 256 there: 6.57 -> 5.53 ms.  (Head dims up to 128, where
// one kernel forms dV and dK: 3.59 -> 3.58 at head dim 72, not worth its code.)
//
// Eight warps: TMA producer, MMA issuer, two idle, four that write the accumulator out.  Every wait is bounded.
struct DkDbSmem {
  static constexpr int kRows = 64, kBox = kRows * 128;      // 64 rows x 64 columns x 2 bytes
  static constexpr int kA = 2 * kBox, kB = 4 * kBox;        // dB and Q of a stage
  static constexpr int kStage = kA + kB, kStages = 2;
  static constexpr int kBars = kStages * kStage;
  static constexpr int bFull = 0, bEmpty = kStages, bDone = 2 * kStages, bCount = 2 * kStages + 1;
  static constexpr int kTmemSlot = kBars + bCount * 8;
  static constexpr int kAbort = kTmemSlot + 8;
  static constexpr int kUsed = kAbort + 8;
  static constexpr int kDynamic = kUsed + 1024;
};
static_assert(2 * (DkDbSmem::kDynamic + 1024) <= 233472, "two CTAs per SM");
constexpr int kDkDbThreads = 256;

// grid = (cdiv(max_sk, 128), Hk, batch)
template <typename T>
__global__ void __launch_bounds__(kDkDbThreads, 2)
sm100_bwd_dk_db_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap tm_db,
                       const __grid_constant__ CUtensorMap tm_q, unsigned int* status) {
  wait_for_earlier_grids();
  using L = DkDbSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kTmemSlot);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kAbort);
  constexpr uint32_t kCols = 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile unsigned int*>(status) != 0u)) return;
  const int z = blockIdx.z, hk = blockIdx.y, n0 = (int)blockIdx.x * kBlk;
  const Seq sq = resolve_seq(p, z);
  if (n0 >= sq.sk) return;
  int m_lo, m_hi;
  query_range(p, sq, n0, min(n0 + kBlk, sq.sk) - 1, m_lo, m_hi);
  if (m_hi < m_lo) {      // keys no query attends to
    zero_rows<T>(p.dk, sq.bidx, hk, sq.k0, n0, sq.sk, p.dqk);
    return;
  }
  const int mb_lo = m_lo / L::kRows, nmb = m_hi / L::kRows - mb_lo + 1;
  const int niter = nmb * p.group;
  const int qboxes = (p.dqk + 63) >> 6;

  if (threadIdx.x == 0) {
    init_abort_and_limit(abort_flag, p.wait_limit_kcycles);
    for (int s = 0; s < L::kStages; ++s) {
      mbar_init(&bars[L::bFull + s], 1);
      mbar_init(&bars[L::bEmpty + s], 1);
    }
    mbar_init(&bars[L::bDone], 1);
    fence_barrier_init();
    prefetch_tmap(&tm_db); prefetch_tmap(&tm_q);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int i = 0, hg = 0, mb = 0; i < niter; ++i) {      // hg, mb: i / nmb, i % nmb
        const int s = i % L::kStages;
        const int h = hk * p.group + hg, row = (mb_lo + mb) * L::kRows;
        if (++mb == nmb) { mb = 0; ++hg; }
        if (!mbar_wait(&bars[L::bEmpty + s], ((uint32_t)(i / L::kStages) & 1u) ^ 1u, abort_flag, status, 0x4000)) break;
        if (p.drop_copy == 4 && i == 0) continue;      // (test hook: the first stage never arrives)
        uint8_t* a = smem + s * L::kStage;
        mbar_expect_tx(&bars[L::bFull + s], L::kA + qboxes * L::kBox);
        for (int b = 0; b < 2; ++b) tma_load_4d(a + b * L::kBox, &tm_db, &bars[L::bFull + s], n0 + b * 64, row, h, sq.bidx);
        for (int b = 0; b < qboxes; ++b)
          tma_load_4d(a + L::kA + b * L::kBox, &tm_q, &bars[L::bFull + s], b * 64, row, h, sq.bidx);
        issued = i + 1;
      }
      if (*abort_flag) {      // copies still in flight land before the CTA gives its shared memory back
        for (int i = max(p.drop_copy == 4 ? 1 : 0, issued - L::kStages); i < issued; ++i)
          mbar_wait_quiet(&bars[L::bFull + i % L::kStages], (uint32_t)(i / L::kStages) & 1u, abort_flag);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_f16(Fmt<T>::code, 128, (uint32_t)((p.dqk + 15) & ~15), 1, 1);
    const uint64_t a_mn = smem_desc_sw128(smem_u32(smem), L::kBox, 1024);
    const uint64_t b_mn = smem_desc_sw128(smem_u32(smem + L::kA), L::kBox, 1024);
    bool ok = true;
    for (int i = 0; ok && i < niter; ++i) {
      const int s = i % L::kStages;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars[L::bFull + s], (uint32_t)(i / L::kStages) & 1u, abort_flag, status, 0x4100)) != 0;
      if (!ok) break;
      tc_fence_after();
      const uint64_t step = (uint64_t)((uint32_t)s * (uint32_t)(L::kStage >> 4));
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < L::kRows / 16; ++kk)
          mma_ss(tmem_base, a_mn + step + (uint32_t)kk * (2048u >> 4), b_mn + step + (uint32_t)kk * (2048u >> 4), idesc,
                 (i > 0 || kk > 0) ? 1u : 0u);
        mma_commit(&bars[L::bEmpty + s]);
        if (i + 1 == niter) mma_commit(&bars[L::bDone]);
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ---- write-out through the (then idle) stages, so that the global stores are row segments ----
    const int quarter = warp & 3, r = quarter * 32 + lane;
    const bool ok = mbar_wait_relaxed(&bars[L::bDone], 0, abort_flag, status, 0x4200);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      T* dst = reinterpret_cast<T*>(p.dk.ptr) + (int64_t)sq.bidx * p.dk.s[0] + (int64_t)hk * p.dk.s[1] + (sq.k0 + n0) * p.dk.s[2];
      for (int c = 0; c * 32 < p.dqk; ++c) {
        float v[32];
        tmem_ld32f(tmem_base + ((uint32_t)(quarter * 32) << 16) + c * 32, v);
        tmem_wait_ld();
        stage_put32<T>(smem_u32(smem), r, c * 32, v, p.sm_scale, 512);
        __syncwarp();
        warp_copy_out<T, 4>(smem_u32(smem), dst, p.dk.s[2], min(kBlk, sq.sk - n0), p.dqk, quarter * 32, c * 4, lane, 512);
        __syncwarp();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kCols);
  }
}
