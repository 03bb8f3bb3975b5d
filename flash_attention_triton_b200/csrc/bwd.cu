// Causal attention backward for sm_100a.
//
// Replaces _backward_kernel_one_col_block and its launcher
// (src/flash_attention_triton/_triton_kernels_v2.py:192-529 of the reference).  Per
// (KV tile j, Q tile i >= j) the maths is that of lines 312-343 there:
//     S = Q K^T, P = exp(scale*S - lse), dP = dO V^T, dS = P o (dP - delta) * scale,
//     dV += P^T dO, dK += dS^T Q, dQ += dS K.
//
// bwd_dkdv_kernel (one CTA per KV tile) works on the TRANSPOSED score tile; see dkdv_roles.
// bwd_dq_kernel (one CTA per Q tile, deterministic path) recomputes S and dP untransposed and
// accumulates dQ_i over ascending j in tensor memory, so each dQ tile has one owner and one
// summation order.
#include "bwd_roles.cuh"

namespace fa2 {
namespace {

// =========================================================================================
// dK / dV (+ fused dQ) kernel: one CTA per KV tile of one (batch, head); see dkdv_roles.
// =========================================================================================
template <int D, bool BF16, int MODE, int KD, int W>
__global__ void __launch_bounds__(DkdvCfg<D, MODE, W>::kThreads, DkdvCfg<D, MODE, W>::kCtasPerSm)
    bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                    const __grid_constant__ CUtensorMap tdk,
                    const __grid_constant__ CUtensorMap tdv, const __grid_constant__ F32Out dk32,
                    const __grid_constant__ F32Out dv32, int cols, const float* rowstats,
                    const unsigned* tile_amax, float* __restrict__ dq_accum, int N,
                    int Nk, int num_bh, int num_heads, int group, float scale, float scale_log2,
                    int* status) {
  using C = DkdvCfg<D, MODE, W>;
  extern __shared__ __align__(1024) uint8_t smem[];
  // Role index: the producer / MMA group takes hardware warps 0-3 (lowest ids on their
  // schedulers), the compute and reduction groups follow; shifts are multiples of 4, so
  // role % 4 is still the tensor-memory lane quarter of the hardware warp.
  constexpr int kWarps = C::kThreads / 32;
  const int warp = ((threadIdx.x >> 5) + C::kMmaWarp) % kWarps, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {
    if (threadIdx.x == 0) atomicCAS(status, 0, 0x20000 | kBSiteAlign);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int ntiles = (N + 127) >> 7;
  const int nktiles = (Nk + 127) >> 7;
  DkdvItem item;
  const HeadTile ht = grouped_order(blockIdx.x, num_bh, nktiles, group);
  item.jt = ht.rank;  // KV tile; tile 0 has the most Q tiles
  item.bh = ht.bh;
  item.hc = HeadCoord{ht.bh % num_heads, ht.bh / num_heads};
  // Spill mode: tiles of a head are numbered KV tile by KV tile, Q tiles ascending inside.
  item.tile0 = static_cast<size_t>(item.bh) * dstile_count(ntiles, nktiles) + dstile_count(ntiles, item.jt);
  item.tile_amax = tile_amax + static_cast<size_t>(item.bh) * ntiles;

  if (threadIdx.x == 0) {
    dkdv_init_barriers<D, MODE, W>(smem_base + C::kOffBar);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const WaitCtx w{abort_flag, status};
  grid_wait_previous();
  grid_allow_next();

  dkdv_roles<D, BF16, MODE, KD, W>(smem, smem_base, tmem_base, warp, lane, &tq, &tk, &tv, &tdo, &tdk, &tdv,
                            dk32, dv32, cols, rowstats, dq_accum, N, Nk, scale, scale_log2, w, item);

  tc_fence_before();
  __syncthreads();
  if (warp == C::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// =========================================================================================
// dQ kernel (deterministic path): one CTA per Q tile, KV tiles in ascending order
// =========================================================================================
// Pipeline per KV tile j:  S(j) = Q K_j^T lands in score buffer j%2, dP(j) = dO V_j^T in the dP
// columns.  The compute warps turn S into P (registers), read dP, release the dP columns
// (so dP(j+1) can be issued while they still work), write dS(j) as 16-bit pairs over the score
// buffer they just read, and the MMA warp then issues dQ += dS(j) K_j followed by S(j+2) into
// the same buffer.  S(j+1) is already in the other buffer, so the tensor pipe and the compute
// warps overlap instead of alternating.
// Head dims up to 64 walk the KV tiles in steps of 64 rows with two CTAs per SM where bwd_step_rows says so, for the
// reasons given at DkdvCfg; the polynomial's share of the exponentials is that of the dK/dV kernel.
template <int D, int W>
struct DqCfg {
  using T = Tile<D>;
  static constexpr int kW = W;  // rows of a KV tile = score columns of a step
  static_assert(W == 128 || (W == 64 && D <= 64), "bwd_step_rows");
  static constexpr int kCtasPerSm = kW == 64 ? 2 : 1;
  static constexpr int kGroups = 2;           // compute groups of four warps
  static constexpr int kCols = kW / kGroups;  // score columns of a compute thread
  static constexpr int kKvBytes = T::kTileBytes / 128 * kW;
  static constexpr int kKStages = kW == 64 ? 4 : 3;  // K_j is needed by S(j) and, later, by dQ(j)
  static constexpr int kVStages = kW == 64 ? 3 : 2;
  static constexpr int kMmaWarp = 4 * kGroups;
  static constexpr int kThreads = 32 * (kMmaWarp + 4);
  static constexpr int kLoadWarp = kMmaWarp + 1;
  // registers per thread of the producer / compute warps; the launch gives every thread kLaunchRegs
  static constexpr int kLaunchRegs = 65536 / (kThreads * kCtasPerSm) / 8 * 8;
  static constexpr int kProducerRegs = kW == 64 ? 48 : 72;
  static constexpr int kComputeRegs = kW == 64 ? 96 : 208;
  static_assert(128 * kProducerRegs + 128 * kGroups * kComputeRegs <= kThreads * kLaunchRegs,
                "setmaxnreg.inc waits for registers that setmaxnreg.dec has released");
  static constexpr int kOffQ = 0;
  static constexpr int kOffDO = kOffQ + T::kTileBytes;
  static constexpr int kOffK = kOffDO + T::kTileBytes;
  static constexpr int kOffV = kOffK + kKStages * kKvBytes;
  static constexpr int kOffStats = kOffV + kVStages * kKvBytes;  // [256] fp32
  static constexpr int kOffBar = kOffStats + 1024;
  static constexpr int kBarQ = 0;  // Q, dO and rowstats
  static constexpr int kBarKFull = 1;
  static constexpr int kBarKEmpty = kBarKFull + kKStages;
  static constexpr int kBarVFull = kBarKEmpty + kKStages;
  static constexpr int kBarVEmpty = kBarVFull + kVStages;
  static constexpr int kBarSFull = kBarVEmpty + kVStages;  // 2 (one per score buffer)
  static constexpr int kBarDpFull = kBarSFull + 2;
  static constexpr int kBarDpConsumed = kBarDpFull + 1;  // one arrival per compute warp
  // 2, by j%2, one arrival per compute warp.  With S(j+1) in the other score buffer, a warp can be through with
  // step j+1 before another one, held up after it has read dP(j), is through with step j; on one barrier
  // it would arrive in that one's place, or complete a phase that the MMA warp has not looked at yet.
  // Step j+2 needs S(j+2), which needs dQ += dS(j) K_j.
  static constexpr int kBarDsReady = kBarDpConsumed + 1;
  static constexpr int kBarDqDone = kBarDsReady + 2;      // 2: dQ += dS(j) K_j completed, by j%2
  static constexpr int kBarDone = kBarDqDone + 2;
  static constexpr int kNumBars = kBarDone + 1;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static constexpr int kColS = 0;     // score buffers at 0 and kW; dS (16-bit) overwrites them
  static constexpr int kColDp = 2 * kW;
  static constexpr int kColDQ = 3 * kW;
  static constexpr int kTmemCols = 512 / kCtasPerSm;
  static_assert(kColDQ + D <= kTmemCols, "tensor memory of one CTA");
  static_assert(kCtasPerSm * (kSmemBytes + 1024) <= 228 * 1024, "shared memory of one SM");
};

template <int D, bool BF16, int KD, int W>
__global__ void __launch_bounds__(DqCfg<D, W>::kThreads, DqCfg<D, W>::kCtasPerSm)
    bwd_dq_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                  const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                  const __grid_constant__ CUtensorMap tdq, const __grid_constant__ F32Out dq32, int cols,
                  const float* rowstats,
                  const unsigned* tile_amax, int N, int Nk, int num_bh, int num_heads,
                  int group, float scale, float scale_log2, int* status) {
  using C = DqCfg<D, W>;
  using T = Tile<D>;
  constexpr int kCols = C::kCols, kPairs = kCols / 2;
  constexpr uint32_t kHalf = kCols;  // columns between the two groups' halves of dS
  extern __shared__ __align__(1024) uint8_t smem[];
  // Role index: producer / MMA group on hardware warps 0-3, compute groups on 4-11.
  const int warp = ((threadIdx.x >> 5) + C::kMmaWarp) % (C::kThreads / 32), lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {
    if (threadIdx.x == 0) atomicCAS(status, 0, 0x20000 | kBSiteAlign);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  auto bar = [&](int i) { return smem_base + C::kOffBar + 8u * i; };

  const int ntiles = (N + 127) >> 7;
  const HeadTile ht = grouped_order(blockIdx.x, num_bh, ntiles, group);
  const int qt = ntiles - 1 - ht.rank;  // the last Q tile meets the most KV tiles
  const int bh = ht.bh;
  const HeadCoord hc{bh % num_heads, bh / num_heads};
  // KV tiles up to the diagonal, or to the last key (N = query rows, Nk <= N = key rows)
  const int nkv = min((qt + 1) * (128 / W), (Nk + W - 1) / W);

  if (threadIdx.x == 0) {
    mbar_init(bar(C::kBarQ), 1);
    for (int i = 0; i < C::kKStages; ++i) {
      mbar_init(bar(C::kBarKFull + i), 1);
      mbar_init(bar(C::kBarKEmpty + i), 2);  // S(j) (warp X) and dQ(j) (warp Y) both done
    }
    for (int i = 0; i < C::kVStages; ++i) {
      mbar_init(bar(C::kBarVFull + i), 1);
      mbar_init(bar(C::kBarVEmpty + i), 1);
    }
    mbar_init(bar(C::kBarSFull + 0), 1);
    mbar_init(bar(C::kBarSFull + 1), 1);
    mbar_init(bar(C::kBarDpFull), 1);
    mbar_init(bar(C::kBarDpConsumed), 4 * C::kGroups);
    mbar_init(bar(C::kBarDsReady + 0), 4 * C::kGroups);
    mbar_init(bar(C::kBarDsReady + 1), 4 * C::kGroups);
    mbar_init(bar(C::kBarDqDone + 0), 1);
    mbar_init(bar(C::kBarDqDone + 1), 1);
    mbar_init(bar(C::kBarDone), 1);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const WaitCtx w{abort_flag, status};
  grid_wait_previous();
  grid_allow_next();

  if (warp >= C::kMmaWarp) {
    reg_dec<C::kProducerRegs>();
    if (warp == C::kLoadWarp) {
      // TMA producer: whole warp, converged; the elected lane arms barriers and issues copies.
      const uint32_t elected = elect_one();
      if (elected) {
        prefetch_tensormap(&tq);
        prefetch_tensormap(&tk);
        prefetch_tensormap(&tv);
        prefetch_tensormap(&tdo);
        mbar_arrive_expect_tx(bar(C::kBarQ), 2 * T::kTileBytes + 1024);
        for (int ch = 0; ch < T::kChunks; ++ch) {
          tma_load_4d(smem_base + C::kOffQ + ch * T::kChunkTileBytes, &tq, ch * T::kChunkElems,
                      qt * 128, hc, bar(C::kBarQ));
          tma_load_4d(smem_base + C::kOffDO + ch * T::kChunkTileBytes, &tdo, ch * T::kChunkElems,
                      qt * 128, hc, bar(C::kBarQ));
        }
        bulk_load_1d(smem_base + C::kOffStats,
                     rowstats + (static_cast<size_t>(bh) * ntiles + qt) * 256, 1024, bar(C::kBarQ));
      }
      for (int j = 0; j < nkv; ++j) {
        const int ks = j % C::kKStages, kph = (j / C::kKStages) & 1;
        if (!mbar_wait_warp(bar(C::kBarKEmpty + ks), kph ^ 1, w, kBSiteLoadQ)) break;
        if (elected) {
          mbar_arrive_expect_tx(bar(C::kBarKFull + ks), C::kKvBytes);
#pragma unroll
          for (int ch = 0; ch < T::kChunks; ++ch)
            tma_load_4d(smem_base + C::kOffK + ks * C::kKvBytes + ch * (C::kKvBytes / T::kChunks), &tk,
                        ch * T::kChunkElems, j * W, hc, bar(C::kBarKFull + ks));
        }
        const int vs = j % C::kVStages, vph = (j / C::kVStages) & 1;
        if (!mbar_wait_warp(bar(C::kBarVEmpty + vs), vph ^ 1, w, kBSiteLoadDO)) break;
        if (elected) {
          mbar_arrive_expect_tx(bar(C::kBarVFull + vs), C::kKvBytes);
#pragma unroll
          for (int ch = 0; ch < T::kChunks; ++ch)
            tma_load_4d(smem_base + C::kOffV + vs * C::kKvBytes + ch * (C::kKvBytes / T::kChunks), &tv,
                        ch * T::kChunkElems, j * W, hc, bar(C::kBarVFull + vs));
        }
      }
    } else if (warp == C::kMmaWarp) {
      // ------------------------------------------------------------ warp X: dP(j) = dO V_j^T
      // (whole warp converged, the elected lane issues).  The three products of a KV step are
      // issued by three warps (X: dP, Z: S, Y: dQ), so none of them waits behind another
      // one's barrier: dP(j+1) only needs the compute warps to have read dP(j), S(j+2) only
      // needs dQ(j) to have consumed dS(j) (both live in score buffer j%2), dQ(j) only needs
      // dS(j).  The tensor pipe executes whatever is issued first.
      const uint32_t elected = elect_one();
      auto commit = [&](int b) {
        if (elected) mma_commit(bar(b));
      };
      const uint32_t doa = smem_base + C::kOffDO;
      int vs = 0, vph = 0;  // ring position of the next V tile
      bool ok = mbar_wait(bar(C::kBarQ), 0, w, kBSiteMmaQ);
      for (int j = 0; ok && j < nkv; ++j) {
        if (j > 0) {
          // dP columns are free once every compute warp has read dP(j-1)
          if (!(ok = mbar_wait(bar(C::kBarDpConsumed), (j - 1) & 1, w, kBSiteMmaDrain))) break;
          tc_fence_after();
        }
        if (!(ok = mbar_wait(bar(C::kBarVFull + vs), vph, w, kBSiteMmaDO))) break;
        issue_rows_x_rows<D, BF16, W, KD>(elected, tmem_base + C::kColDp, doa,
                                   smem_base + C::kOffV + vs * C::kKvBytes);
        commit(C::kBarDpFull);
        commit(C::kBarVEmpty + vs);  // V is free once dP has read it
        if (++vs == C::kVStages) {
          vs = 0;
          vph ^= 1;
        }
      }
    } else if (warp == C::kMmaWarp + 3) {
      // ------------------------------------------------------------ warp Z: S(j) = Q K_j^T
      const uint32_t elected = elect_one();
      auto commit = [&](int b) {
        if (elected) mma_commit(bar(b));
      };
      const uint32_t qa = smem_base + C::kOffQ;
      int ks = 0, kph = 0;  // ring position of the next K tile
      bool ok = mbar_wait(bar(C::kBarQ), 0, w, kBSiteMmaQ);
      for (int j = 0; ok && j < nkv; ++j) {
        if (j >= 2) {
          // score buffer j%2 holds dS(j-2) until dQ += dS(j-2) K_(j-2) has completed
          if (!(ok = mbar_wait(bar(C::kBarDqDone + (j & 1)), ((j - 2) >> 1) & 1, w, kBSiteMmaDs)))
            break;
          tc_fence_after();
        }
        if (!(ok = mbar_wait(bar(C::kBarKFull + ks), kph, w, kBSiteMmaKV))) break;
        issue_rows_x_rows<D, BF16, W, KD>(elected, tmem_base + C::kColS + (j & 1) * W, qa,
                                   smem_base + C::kOffK + ks * C::kKvBytes);
        commit(C::kBarSFull + (j & 1));
        commit(C::kBarKEmpty + ks);
        if (++ks == C::kKStages) {
          ks = 0;
          kph ^= 1;
        }
      }
    } else if (warp == C::kMmaWarp + 2) {
      // ------------------------------------------------------------ warp Y: dQ += dS(j) K_j
      const uint32_t elected = elect_one();
      auto commit = [&](int b) {
        if (elected) mma_commit(bar(b));
      };
      bool ok = true;
      int ks = 0, kph = 0;
      for (int j = 0; ok && j < nkv; ++j) {
        if (!(ok = mbar_wait(bar(C::kBarKFull + ks), kph, w, kBSiteMmaKV))) break;
        if (!(ok = mbar_wait(bar(C::kBarDsReady + (j & 1)), (j >> 1) & 1, w, kBSiteMmaDs))) break;
        tc_fence_after();
        // A = 16-bit dS over score buffer j%2, B = K_j as MN-major tile
        issue_tmem_x_tile<D, BF16, W, KD>(elected, tmem_base + C::kColDQ, tmem_base + C::kColS + (j & 1) * W,
                                   kHalf, smem_base + C::kOffK + ks * C::kKvBytes, j > 0);
        commit(C::kBarDqDone + (j & 1));
        commit(C::kBarKEmpty + ks);
        if (++ks == C::kKStages) {
          ks = 0;
          kph ^= 1;
        }
      }
      if (ok) commit(C::kBarDone);
    }
    __syncwarp();
  } else {
    reg_inc<C::kComputeRegs>();
    const int wg = warp >> 2;
    const int w4 = warp & 3;
    const int r = w4 * 32 + lane;  // q row in the tile = tensor-memory lane
    const uint32_t lane_base = static_cast<uint32_t>(w4 * 32) << 16;
    const uint32_t tDp = tmem_base + lane_base + C::kColDp + wg * kCols;
    const float2 sc2 = make_float2(scale_log2, scale_log2);
    // dS is formed as dS * 2^k in fp16 and dQ multiplied by 2^-k at the end (head_dscale)
    float inv_dscale;
    const float dscale =
        head_dscale<BF16>(tile_amax + static_cast<size_t>(bh) * ntiles, ntiles, lane, &inv_dscale);
    const float2 scale2 = make_float2(scale * dscale, scale * dscale);
    bool ok = mbar_wait_warp(bar(C::kBarQ), 0, w, kBSiteCmpQ);
    float2 nlse2 = make_float2(0.f, 0.f), ndlt2 = make_float2(0.f, 0.f);
    if (ok) {
      const float* stats = reinterpret_cast<const float*>(smem + C::kOffStats);
      nlse2 = make_float2(stats[r], stats[r]);              // -lse*log2e of this row
      ndlt2 = make_float2(stats[128 + r], stats[128 + r]);  // -delta of this row
    }
    for (int j = 0; ok && j < nkv; ++j) {
      const uint32_t tS = tmem_base + lane_base + C::kColS + (j & 1) * W + wg * kCols;
      if (!(ok = mbar_wait_warp(bar(C::kBarSFull + (j & 1)), (j >> 1) & 1, w, kBSiteCmpSt))) break;
      tc_fence_after();
      float2 p[kPairs];
      {
        uint32_t sr[kCols];
#pragma unroll
        for (int c = 0; c < kCols; c += 32) tmem_ld_x32(tS + c, sr + c);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kPairs; ++c) {
          const float2 t = __ffma2_rn(
              make_float2(__uint_as_float(sr[2 * c]), __uint_as_float(sr[2 * c + 1])), sc2, nlse2);
          p[c] = exp2_pair<kPolyShareT<D>>(t, c);
        }
      }
      if (j * W + W > qt * 128 || j * W + W > Nk) {
        // diagonal tiles: keep kv <= q; last KV tile: drop the columns beyond the last key
        const int last = min(qt * 128 + r, Nk - 1) - j * W - wg * kCols;
#pragma unroll
        for (int c = 0; c < kPairs; ++c) {
          p[c].x = (2 * c <= last) ? p[c].x : 0.f;
          p[c].y = (2 * c + 1 <= last) ? p[c].y : 0.f;
        }
      }
      if (!(ok = mbar_wait_warp(bar(C::kBarDpFull), j & 1, w, kBSiteCmpDpt))) break;
      tc_fence_after();
      uint32_t dp[kCols];
#pragma unroll
      for (int c = 0; c < kCols; c += 32) tmem_ld_x32(tDp + c, dp + c);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarDpConsumed));
      uint32_t dsk[kPairs];
#pragma unroll
      for (int c = 0; c < kPairs; ++c) {
        float2 u = __fadd2_rn(
            make_float2(__uint_as_float(dp[2 * c]), __uint_as_float(dp[2 * c + 1])), ndlt2);
        u = __fmul2_rn(__fmul2_rn(p[c], u), scale2);
        dsk[c] = pack2<kInterBF16<BF16>>(u.x, u.y);
      }
      // over the score columns this thread has already read
      if constexpr (kPairs == 16) tmem_st_x16(tS, dsk); else tmem_st_x32(tS, dsk);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarDsReady + (j & 1)));
    }
    if (ok && wg == 0 && mbar_wait_warp(bar(C::kBarDone), 0, w, kBSiteCmpDone)) {
      tc_fence_after();
      if (dq32.p != nullptr)
        store_rows_f32<KD>(tmem_base + lane_base + C::kColDQ, dq32, cols, qt * 128 + r, hc, N, inv_dscale);
      else
        store_rows_16bit<D, BF16, KD>(tmem_base + lane_base + C::kColDQ, smem + C::kOffDO, w4, lane, &tdq,
                                qt * 128, hc, N, inv_dscale);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == C::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// =========================================================================================
// One output tile per CTA from spilled 16-bit tiles (head dim 256: dK and dQ; see
// consume_roles).  warps 0-3 epilogue, warp 4 producer, warp 5 MMA issue.
// =========================================================================================
// Up to head dim 128 two CTAs run on an SM (rings of three 32 KiB stages at head dim 128).  With one,
// the SM reads nothing while its CTA sets up (tensor memory, barriers, first loads) and stores its
// result, some 6 us beside the few products of a short sum; two cover each other.  Whole backward,
// microseconds, one CTA with whole tiles against two: [2,32,8192,128] bf16 3105 -> 2971, [32,20,1024,96]
// fp16 868 -> 786, [1,32,4096,128] 467 -> 438, [8,32,512,128] 143 -> 133, [1,2,32768,128] 1409 / 1431 ->
// 1450 / 1343 in two runs; three CTAs with two stages each measured the same within 1 %.
template <int D>
struct ConsumeCfg {
  using T = Tile<D>;
  static constexpr int kCtasPerSm = D == 256 ? 1 : 2;
  static constexpr int kThreads = 192;
  static constexpr int kLoadWarp = 4;
  static constexpr int kMmaWarp = 5;
  // scratch tile, then the operand tile (halves of them up to head dim 128)
  static constexpr int kStageBytes = (32768 + T::kTileBytes) / consume_parts(D);
  static constexpr int kStages = (228 * 1024 / kCtasPerSm - 2048) / kStageBytes;
  static constexpr int kOffBar = kStages * kStageBytes;
  static constexpr int kNumBars = 2 * kStages + 1;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static constexpr int kTmemCols = D < 32 ? 32 : D;
  static_assert(kSmemBytes <= 232448 && kCtasPerSm * (kSmemBytes + 1024) <= 228 * 1024, "shared memory");
  static_assert(kStages * kStageBytes >= T::kTileBytes, "the ring stages the output at the end");
};

template <int D, bool BF16, int FORM, int KD = D>
__global__ void __launch_bounds__(ConsumeCfg<D>::kThreads, ConsumeCfg<D>::kCtasPerSm)
    bwd_consume_kernel(const uint4* scratch, const __grid_constant__ CUtensorMap tb,
                       const __grid_constant__ CUtensorMap tout, const __grid_constant__ F32Out out32, int cols,
                       const unsigned* tile_amax, int N, int Nk, int num_bh,
                       int num_heads, int group, int* status) {
  using C = ConsumeCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {
    if (threadIdx.x == 0) atomicCAS(status, 0, 0x20000 | kBSiteAlign);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int ntiles = (N + 127) >> 7;     // Q tiles
  const int nktiles = (Nk + 127) >> 7;   // KV tiles
  ConsumeItem item;
  const HeadTile ht = grouped_order(blockIdx.x, num_bh, FORM == 2 ? ntiles : nktiles, group);
  const int bh = ht.bh;
  item.hc = HeadCoord{bh % num_heads, bh / num_heads};
  item.head_tile0 = static_cast<size_t>(bh) * dstile_count(ntiles, nktiles);
  // the last Q tile (form 2) and the first KV tile (form 1) are summed over the most tiles
  item.ot = FORM == 2 ? ntiles - 1 - ht.rank : ht.rank;
  item.tile_amax = tile_amax + static_cast<size_t>(bh) * ntiles;

  if (threadIdx.x == 0) {
    consume_init_barriers<C::kStages>(smem_base + C::kOffBar);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const WaitCtx w{abort_flag, status};
  grid_wait_previous();
  grid_allow_next();

  consume_roles<D, BF16, FORM, C::kStages, KD>(smem, smem_base, smem_base + C::kOffBar, tmem_base,
                                           warp == C::kLoadWarp, warp == C::kMmaWarp,
                                           warp < 4 ? warp : -1, lane, scratch, &tb, &tout, out32, cols, N, Nk, w,
                                           item);

  tc_fence_before();
  __syncthreads();
  if (warp == C::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

// =========================================================================================
// The same for two adjacent output tiles of head dim 256 per CTA.  One tile per CTA reads 32 KiB of
// scratch and 64 KiB of operand for every 1024 cycles of tensor work, and the L2 cannot deliver 96 KiB
// an SM in that time (2 000 - 2 175 cycles measured); two tiles share the operand, 64 KiB a product,
// and come close to what reading the scratch from HBM takes.  Both accumulators fill the tensor
// memory.  Shared memory: a ring of two stages of both scratch tiles (64 KiB each) and a ring of three
// half operand tiles (64 reduction rows, 32 KiB each).  Every output tile adds the same products in the
// same order as above, so the two kernels give the same bits.
// warps 0-3 and 4-7 epilogue of the first and the second tile, warp 8 producer, warp 9 MMA issue.
// Measured on the whole backward, bf16, one tile a CTA -> two: [1,32,8192,256] 2690 -> 2542 us, [1,32,8192,192] 2394 -> 2179.
// =========================================================================================
struct ConsumePairCfg {
  using T = Tile<256>;
  static constexpr int kThreads = 320;
  static constexpr int kLoadWarp = 8;
  static constexpr int kMmaWarp = 9;
  static constexpr int kAStages = 2, kAStageBytes = 2 * 32768;
  static constexpr int kBStages = 3, kBStageBytes = T::kTileBytes / 2;
  static constexpr int kOffA = 0;
  static constexpr int kOffB = kAStages * kAStageBytes;
  static constexpr int kOffBar = kOffB + kBStages * kBStageBytes;
  static constexpr int kBarAFull = 0;
  static constexpr int kBarAEmpty = kBarAFull + kAStages;
  static constexpr int kBarBFull = kBarAEmpty + kAStages;
  static constexpr int kBarBEmpty = kBarBFull + kBStages;
  static constexpr int kBarDone = kBarBEmpty + kBStages;
  static constexpr int kNumBars = kBarDone + 1;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 232448, "shared memory budget of one CTA");
  static_assert(kAStages * kAStageBytes >= 2 * T::kTileBytes, "the scratch ring stages both outputs at the end");
};

template <bool BF16, int FORM, int KD>
__global__ void __launch_bounds__(ConsumePairCfg::kThreads, 1)
    bwd_consume_pair_kernel(const uint4* scratch, const __grid_constant__ CUtensorMap tb,
                            const __grid_constant__ CUtensorMap tout, const __grid_constant__ F32Out out32,
                            int cols, const unsigned* tile_amax, int N, int Nk, int num_bh,
                            int num_heads, int group, int* status) {
  using C = ConsumePairCfg;
  using T = Tile<256>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {
    if (threadIdx.x == 0) atomicCAS(status, 0, 0x20000 | kBSiteAlign);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  auto bar = [&](int i) { return smem_base + C::kOffBar + 8u * i; };

  const int ntiles = (N + 127) >> 7;    // Q tiles
  const int nktiles = (Nk + 127) >> 7;  // KV tiles
  const int out_tiles = FORM == 2 ? ntiles : nktiles;
  const int out_rows = FORM == 2 ? N : Nk;
  const int npairs = (out_tiles + 1) >> 1;
  const HeadTile ht = grouped_order(blockIdx.x, num_bh, npairs, group);
  const int bh = ht.bh;
  const HeadCoord hc{bh % num_heads, bh / num_heads};
  const size_t head_tile0 = static_cast<size_t>(bh) * dstile_count(ntiles, nktiles);
  // the last Q tiles (form 2) and the first KV tiles (form 1) are summed over the most tiles
  const int ot0 = 2 * (FORM == 2 ? npairs - 1 - ht.rank : ht.rank);
  // Range of tiles of the other kind each output tile is summed over: [begin, end).  Both start at 0
  // (form 2) or both end at ntiles (form 1); a missing second tile has an empty range.
  int begin[2], end[2];
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    const int ot = ot0 + o;
    begin[o] = FORM == 2 ? 0 : ot;
    end[o] = ot >= out_tiles ? begin[o] : (FORM == 2 ? min(ot + 1, nktiles) : ntiles);
  }
  const int first = begin[0], last = max(end[0], end[1]);
  auto wanted = [&](int o, int x) { return x >= begin[o] && x < end[o]; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kNumBars; ++i) mbar_init(bar(i), 1);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const WaitCtx w{abort_flag, status};
  grid_wait_previous();
  grid_allow_next();

  if (warp == C::kLoadWarp) {
    const uint32_t elected = elect_one();
    if (elected) prefetch_tensormap(&tb);
    bool ok = true;
    for (int x = first, n = 0; ok && x < last; ++x, ++n) {
      const int st = n % C::kAStages, ph = (n / C::kAStages) & 1;
      if (!(ok = mbar_wait_warp(bar(C::kBarAEmpty + st), ph ^ 1, w, kBSiteLoadQ))) break;
      if (elected) {
        mbar_arrive_expect_tx(bar(C::kBarAFull + st), 32768u * (wanted(0, x) + wanted(1, x)));
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          if (!wanted(o, x)) continue;
          const int jt = FORM == 2 ? x : ot0 + o, qt = FORM == 2 ? ot0 + o : x;
          const size_t tile = head_tile0 + dstile_count(ntiles, jt) + (qt - jt);
          bulk_load_1d(smem_base + C::kOffA + st * C::kAStageBytes + o * 32768, scratch + tile * 2048, 32768,
                       bar(C::kBarAFull + st));
        }
      }
      for (int half = 0; half < 2; ++half) {
        const int m = 2 * n + half, bs = m % C::kBStages, bph = (m / C::kBStages) & 1;
        if (!(ok = mbar_wait_warp(bar(C::kBarBEmpty + bs), bph ^ 1, w, kBSiteLoadDO))) break;
        if (elected) {
          mbar_arrive_expect_tx(bar(C::kBarBFull + bs), C::kBStageBytes / T::kChunks * (KD / T::kChunkElems));
#pragma unroll
          for (int ch = 0; ch < KD / T::kChunkElems; ++ch)
            tma_load_4d(smem_base + C::kOffB + bs * C::kBStageBytes + ch * (C::kBStageBytes / T::kChunks), &tb,
                        ch * T::kChunkElems, x * 128 + half * 64, hc, bar(C::kBarBFull + bs));
        }
      }
    }
    __syncwarp();
  } else if (warp == C::kMmaWarp) {
    const uint32_t elected = elect_one();
    bool ok = true;
    for (int x = first, n = 0; ok && x < last; ++x, ++n) {
      const int st = n % C::kAStages, ph = (n / C::kAStages) & 1;
      if (!(ok = mbar_wait(bar(C::kBarAFull + st), ph, w, kBSiteMmaKV))) break;
      for (int half = 0; half < 2; ++half) {
        const int m = 2 * n + half, bs = m % C::kBStages, bph = (m / C::kBStages) & 1;
        if (!(ok = mbar_wait(bar(C::kBarBFull + bs), bph, w, kBSiteMmaQ))) break;
#pragma unroll
        for (int o = 0; o < 2; ++o)
          if (wanted(o, x))
            issue_pieces_x_half_tile<256, BF16, FORM == 2, KD>(
                elected, tmem_base + o * 256, smem_base + C::kOffA + st * C::kAStageBytes + o * 32768, half,
                smem_base + C::kOffB + bs * C::kBStageBytes, half > 0 || x > begin[o]);
        if (elected) mma_commit(bar(C::kBarBEmpty + bs));
      }
      if (ok && elected) mma_commit(bar(C::kBarAEmpty + st));
    }
    if (ok && elected) mma_commit(bar(C::kBarDone));
    __syncwarp();
  } else {
    const int o = warp >> 2, w4 = warp & 3, ot = ot0 + o;
    float inv_dscale;  // dS tiles carry the head's power-of-two factor
    head_dscale<BF16>(tile_amax + static_cast<size_t>(bh) * ntiles, ntiles, lane, &inv_dscale);
    if (mbar_wait_warp(bar(C::kBarDone), 0, w, kBSiteCmpDone) && ot < out_tiles) {
      tc_fence_after();
      const uint32_t acc = tmem_base + o * 256 + (static_cast<uint32_t>(w4 * 32) << 16);
      if (out32.p != nullptr)
        store_rows_f32<KD>(acc, out32, cols, ot * 128 + w4 * 32 + lane, hc, out_rows, inv_dscale);
      else  // every product has completed, so the scratch ring is idle
        store_rows_16bit<256, BF16, KD>(acc, smem + C::kOffA + o * T::kTileBytes, w4, lane, &tout, ot * 128, hc,
                                    out_rows, inv_dscale);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == C::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// =========================================================================================
// Head dims above 128: scores and dV.  dK and dV together would fill the 512 tensor-memory columns, so
// the backward is split: this kernel forms P^T and dS^T for every (KV tile, Q tile) pair, accumulates
// dV += P^T dO in tensor memory and writes dS^T as 16-bit piece-major tiles to a scratch tensor;
// bwd_consume_kernel then forms dK and dQ from them.  CTA = one KV tile.  K and V stay in shared memory as
// kChunks chunk tiles of 64 columns each (128 KiB together at head dim 256); Q and dO stream through a ring of six such
// chunks (eight up to head dim 192), in the order Q(i), dO(i), Q(i+1), ...; dO(i) keeps its chunks until dV has been formed
// with them, which leaves two (five) for what comes next.  Tensor memory: St, dPt (128 columns each), dV (256).
//   warps 0-7  compute (as in bwd_dkdv_kernel: kv row per thread, two groups of 64 q columns)
//   warp  8    MMA issue, per step:  [Pt(i) ready]  dV += Pt(i) dO(i),  St(i+1) = K Q^T (over Pt(i)),
//              [dPt(i) copied]  dPt(i+1) = V dO^T.  dPt(i+1) runs under the exponentials of St(i+1).
//   warp  9    TMA producer
// Bound by the chain of a step: ncu ([1,16,8192,256] bf16) has the tensor pipe at 66 % of the active cycles (4 660 a pair, 3 072 of
// them tensor, 3 584 shared-memory time), L1 at 55 %, DRAM at 24 %; without the ring's loads 6 % less, without the dS stores
// 12 %.  In a loop of long sequences the power limit takes the clock from 1.5 to 1.25 GHz besides.  The version before
// wrote P^T to a second scratch tensor too, from which a third consumer formed dV: 4.4 of 10.9 GB on
// [2,16,8192,256] bf16, forward and backward 4 148 -> 3 690 us in a loop.  Same bits.  Walking the Q tiles
// from the last one, as bwd_dkdv_kernel does, measured the same.
// =========================================================================================
template <int N>
struct Columns {
  static constexpr int value = N;
};

template <int CH>
struct ScoresCfg {
  using T = Tile<128>;
  static constexpr int kThreads = 384;
  static constexpr int kMmaWarp = 8;
  static constexpr int kLoadWarp = 9;
  static constexpr int kChunks = CH;  // of 64 columns: 4 at head dim 256, 3 up to 192
  static constexpr int kChunkBytes = T::kChunkTileBytes;
  static constexpr int kRing = 14 - 2 * CH;
  static constexpr int kOffK = 0;
  static constexpr int kOffV = kChunks * kChunkBytes;
  static constexpr int kOffRing = 2 * kChunks * kChunkBytes;
  static constexpr int kOffStats = kOffRing + kRing * kChunkBytes;  // [2][256] fp32
  static constexpr int kOffBar = kOffStats + 2 * 1024;
  static constexpr int kBarKV = 0;
  static constexpr int kBarRingFull = 1;
  static constexpr int kBarRingEmpty = kBarRingFull + kRing;
  static constexpr int kBarStFull = kBarRingEmpty + kRing;
  static constexpr int kBarPtReady = kBarStFull + 1;     // 8 arrivals
  static constexpr int kBarDptFull = kBarPtReady + 1;
  static constexpr int kBarDptFree = kBarDptFull + 1;    // 8 arrivals
  static constexpr int kBarStatsFull = kBarDptFree + 1;  // 2
  static constexpr int kBarStatsFree = kBarStatsFull + 2;  // 2, 8 arrivals
  static constexpr int kBarDone = kBarStatsFree + 2;
  static constexpr int kNumBars = kBarDone + 1;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 232448, "shared memory budget of one CTA");
  static constexpr int kColSt = 0;  // Pt(i) is written over St(i)
  static constexpr int kColDpt = 128;
  static constexpr int kColDV = 256;
  static constexpr int kTmemCols = 512;
};

template <bool BF16, int CH>
__global__ void __launch_bounds__(ScoresCfg<CH>::kThreads, 1)
    bwd_scores_wide_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                           const __grid_constant__ CUtensorMap tv,
                           const __grid_constant__ CUtensorMap tdo, const __grid_constant__ CUtensorMap tdv,
                           const __grid_constant__ F32Out dv32, int cols, const float* rowstats,
                           const unsigned* tile_amax, uint4* __restrict__ ds_scratch, int N, int Nk, int num_bh,
                           int num_heads, int group, float scale, float scale_log2, int* status) {
  using C = ScoresCfg<CH>;
  using T = Tile<128>;
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int kWarps = C::kThreads / 32;
  const int warp = ((threadIdx.x >> 5) + C::kMmaWarp) % kWarps, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {
    if (threadIdx.x == 0) atomicCAS(status, 0, 0x20000 | kBSiteAlign);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  auto bar = [&](int i) { return smem_base + C::kOffBar + 8u * i; };

  const int ntiles = (N + 127) >> 7;
  const int nktiles = (Nk + 127) >> 7;
  const HeadTile ht = grouped_order(blockIdx.x, num_bh, nktiles, group);
  const int jt = ht.rank;  // KV tile
  const int bh = ht.bh;
  const HeadCoord hc{bh % num_heads, bh / num_heads};
  const int nq = ntiles - jt;  // Q tiles jt .. ntiles-1
  const bool kv_ragged = jt * 128 + 128 > Nk;
  const int tile0 = bh * dstile_count(ntiles, nktiles) + dstile_count(ntiles, jt);

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kNumBars; ++i) {
      const bool compute = i == C::kBarPtReady || i == C::kBarDptFree || i == C::kBarStatsFree || i == C::kBarStatsFree + 1;
      mbar_init(bar(i), compute ? 8 : 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const WaitCtx w{abort_flag, status};
  grid_wait_previous();
  grid_allow_next();

  if (warp >= C::kMmaWarp) {
    reg_dec<72>();
    if (warp == C::kLoadWarp) {
      const uint32_t elected = elect_one();
      if (elected) {
        prefetch_tensormap(&tq);
        prefetch_tensormap(&tk);
        prefetch_tensormap(&tv);
        prefetch_tensormap(&tdo);
        mbar_arrive_expect_tx(bar(C::kBarKV), 2 * C::kChunks * C::kChunkBytes);
        for (int ch = 0; ch < C::kChunks; ++ch) {
          tma_load_4d(smem_base + C::kOffK + ch * C::kChunkBytes, &tk, ch * T::kChunkElems, jt * 128, hc, bar(C::kBarKV));
          tma_load_4d(smem_base + C::kOffV + ch * C::kChunkBytes, &tv, ch * T::kChunkElems, jt * 128, hc, bar(C::kBarKV));
        }
      }
      bool ok = true;
      int slot = 0, ph = 0;
      for (int i = 0; ok && i < nq; ++i) {
        const int qt = jt + i;
        // rowstats of Q tile qt -> stats buffer i % 2, once the compute warps are done with
        // tile i - 2
        if (!(ok = mbar_wait_warp(bar(C::kBarStatsFree + (i & 1)), ((i >> 1) & 1) ^ 1, w, kBSiteLoadQ)))
          break;
        if (elected) {
          mbar_arrive_expect_tx(bar(C::kBarStatsFull + (i & 1)), 1024);
          bulk_load_1d(smem_base + C::kOffStats + (i & 1) * 1024,
                       rowstats + (static_cast<size_t>(bh) * ntiles + qt) * 256, 1024,
                       bar(C::kBarStatsFull + (i & 1)));
        }
        for (int sub = 0; sub < 2 * C::kChunks; ++sub) {  // the chunks of Q, then those of dO
          if (!(ok = mbar_wait_warp(bar(C::kBarRingEmpty + slot), ph ^ 1, w, kBSiteLoadDO))) break;
          if (elected) {
            mbar_arrive_expect_tx(bar(C::kBarRingFull + slot), C::kChunkBytes);
            tma_load_4d(smem_base + C::kOffRing + slot * C::kChunkBytes, sub < C::kChunks ? &tq : &tdo,
                        (sub % C::kChunks) * T::kChunkElems, qt * 128, hc, bar(C::kBarRingFull + slot));
          }
          if (++slot == C::kRing) slot = 0, ph ^= 1;
        }
      }
    } else if (warp == C::kMmaWarp) {
      const uint32_t elected = elect_one();
      auto commit = [&](int b) {
        if (elected) mma_commit(bar(b));
      };
      bool ok = mbar_wait(bar(C::kBarKV), 0, w, kBSiteMmaKV);
      int slot = 0, ph = 0;  // of the next chunk
      // St and dPt: 64 columns of the head dim after another, from the next chunks of the ring
      auto scores = [&](int column, int resident, bool release) {
        for (int ch = 0; ok && ch < C::kChunks; ++ch) {
          if (!(ok = mbar_wait(bar(C::kBarRingFull + slot), ph, w, kBSiteMmaQ))) break;
          issue_rows_x_rows<64, BF16>(elected, tmem_base + column, smem_base + resident + ch * C::kChunkBytes,
                                      smem_base + C::kOffRing + slot * C::kChunkBytes, ch > 0);
          if (release) commit(C::kBarRingEmpty + slot);
          if (++slot == C::kRing) slot = 0, ph ^= 1;
        }
      };
      for (int i = 0; ok && i <= nq; ++i) {
        if (i > 0) {
          int s = (slot + C::kRing - C::kChunks) % C::kRing;  // dO(i-1) lies in the last chunks taken
          if (!(ok = mbar_wait(bar(C::kBarPtReady), (i - 1) & 1, w, kBSiteMmaPt))) break;
          tc_fence_after();
          for (int ch = 0; ch < C::kChunks; ++ch) {
            issue_tmem_x_tile<64, BF16>(elected, tmem_base + C::kColDV + ch * 64, tmem_base + C::kColSt, 64,
                                        smem_base + C::kOffRing + s * C::kChunkBytes, i > 1);
            commit(C::kBarRingEmpty + s);
            if (++s == C::kRing) s = 0;
          }
        }
        if (i == nq) break;
        scores(C::kColSt, C::kOffK, true);
        if (!ok) break;
        commit(C::kBarStFull);
        if (i > 0) {
          if (!(ok = mbar_wait(bar(C::kBarDptFree), (i - 1) & 1, w, kBSiteMmaDrain))) break;
          tc_fence_after();
        }
        scores(C::kColDpt, C::kOffV, false);
        if (ok) commit(C::kBarDptFull);
      }
      if (ok) commit(C::kBarDone);
    }
    __syncwarp();
  } else {
    reg_inc<208>();
    const int wg = warp >> 2;  // 0: q columns 0..63 of the tile, 1: 64..127
    const int w4 = warp & 3;
    const int r = w4 * 32 + lane;  // kv row in the tile = tensor-memory lane
    const uint32_t lane_base = static_cast<uint32_t>(w4 * 32) << 16;
    const uint32_t tSt = tmem_base + lane_base + C::kColSt + wg * 64;
    const uint32_t tDpt = tmem_base + lane_base + C::kColDpt + wg * 64;
    const float2 sc2 = make_float2(scale_log2, scale_log2);
    float inv_dscale;
    const float dscale =
        head_dscale<BF16>(tile_amax + static_cast<size_t>(bh) * ntiles, ntiles, lane, &inv_dscale);
    const float2 scale2 = make_float2(scale * dscale, scale * dscale);  // dS * 2^k, see head_dscale
    bool ok = true;
    for (int i = 0; i < nq; ++i) {
      const int b = i & 1;
      const float* stats = reinterpret_cast<const float*>(smem + C::kOffStats + b * 1024);
      const float4* nlse = reinterpret_cast<const float4*>(stats + wg * 64);        // -lse*log2e
      const float4* ndlt = reinterpret_cast<const float4*>(stats + 128 + wg * 64);  // -delta
      if (!(ok = mbar_wait_warp(bar(C::kBarStatsFull + b), (i >> 1) & 1, w, kBSiteCmpQ))) break;
      if (!(ok = mbar_wait_warp(bar(C::kBarStFull), i & 1, w, kBSiteCmpSt))) break;
      tc_fence_after();
      float2 p[32];  // P^T for this thread's kv row, q columns wg*64 .. wg*64+63
      {
        uint32_t sr[64];
        tmem_ld_x32(tSt, sr);
        tmem_ld_x32(tSt + 32, sr + 32);
        tmem_wait_ld();
        probabilities_of_row(sr, nlse, sc2, p);
      }
      if (i == 0 || kv_ragged) {
        // diagonal tile: keep q >= kv; rows beyond the last key keep nothing
        mask_row(p, (jt * 128 + r >= Nk) ? 128 : (i == 0 ? r : 0), wg * 64);
      }
      {
        uint32_t pk[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) pk[c] = pack2<kInterBF16<BF16>>(p[c].x, p[c].y);
        tmem_st_x32(tSt, pk);
        tmem_wait_st();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarPtReady));

      if (!(ok = mbar_wait_warp(bar(C::kBarDptFull), i & 1, w, kBSiteCmpDpt))) break;
      tc_fence_after();
      uint32_t dp[64];
      tmem_ld_x32(tDpt, dp);
      tmem_ld_x32(tDpt + 32, dp + 32);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarDptFree));
      uint32_t dsk[32];
#pragma unroll
      for (int c4 = 0; c4 < 16; ++c4) {
        const float4 nd = ndlt[c4];
        // dS = P * (dP - delta) * scale, scale folded in before the 16-bit rounding
        float2 u0 = __fadd2_rn(make_float2(__uint_as_float(dp[4 * c4]), __uint_as_float(dp[4 * c4 + 1])),
                               make_float2(nd.x, nd.y));
        float2 u1 = __fadd2_rn(make_float2(__uint_as_float(dp[4 * c4 + 2]), __uint_as_float(dp[4 * c4 + 3])),
                               make_float2(nd.z, nd.w));
        u0 = __fmul2_rn(__fmul2_rn(p[2 * c4], u0), scale2);
        u1 = __fmul2_rn(__fmul2_rn(p[2 * c4 + 1], u1), scale2);
        dsk[2 * c4] = pack2<kInterBF16<BF16>>(u0.x, u0.y);
        dsk[2 * c4 + 1] = pack2<kInterBF16<BF16>>(u1.x, u1.y);
      }
      {
        // piece-major, see bwd_dkdv_kernel's spill store
        uint4* dst = ds_scratch + (static_cast<size_t>(tile0 + i) * 2048 + wg * 1024 + r);
#pragma unroll
        for (int pc = 0; pc < 8; ++pc)
          dst[pc * 128] = make_uint4(dsk[4 * pc], dsk[4 * pc + 1], dsk[4 * pc + 2], dsk[4 * pc + 3]);
      }
      // The row statistics are given back only after the stores of the values computed from them:
      // an arrive that merely follows the loads in program order can overtake the last of them, and
      // the copy engine then refills the buffer under it (seen as four wrong q columns of a tile).
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarStatsFree + b));
    }
    // dV: group 0 stores columns 0..127, group 1 the others, staged through the idle K tile
    if (ok && mbar_wait_warp(bar(C::kBarDone), 0, w, kBSiteCmpDone)) {
      tc_fence_after();
      const uint32_t acc = tmem_base + lane_base + C::kColDV + wg * 128;
      auto store = [&](auto columns) {
        if (dv32.p != nullptr)
          store_rows_f32<columns.value>(acc, F32Out{dv32.p + wg * 128, dv32.st}, cols - wg * 128, jt * 128 + r, hc, Nk);
        else
          store_rows_16bit<128, BF16, columns.value>(acc, smem + C::kOffK + wg * T::kTileBytes, w4, lane, &tdv, jt * 128, hc,
                                                     Nk, 1.0f, wg * T::kChunks);
      };
      if (wg == 0) store(Columns<128>{}); else store(Columns<CH * 64 - 128>{});
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == C::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <bool BF16, int CH>
cudaError_t launch_scores_wide_t(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                                 const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdv,
                                 const F32Out& dv32, const RowStats& rowstats, void* ds_scratch, int* status,
                                 cudaStream_t stream) {
  using C = ScoresCfg<CH>;
  auto kern = bwd_scores_wide_kernel<BF16, CH>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const unsigned grid = static_cast<unsigned>((s.Nk + 127) / 128) * s.B * s.H;  // one CTA per KV tile
  return launch_dependent(kern, grid, C::kThreads, C::kSmemBytes, stream,
      tq, tk, tv, tdo, tdv, dv32, s.Dg, rowstats.stats, rowstats.tile_amax, static_cast<uint4*>(ds_scratch), s.N, s.Nk, s.B * s.H, s.H, heads_per_group(s), s.scale,
      s.scale * 1.4426950408889634f, status);
}

template <int D, bool BF16, int MODE, int KD = D, int W = 128>
cudaError_t launch_dkdv_t(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                          const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdk,
                          const CUtensorMap& tdv, const F32Out& dk32, const F32Out& dv32,
                          const RowStats& rowstats, float* dq_accum,
                          int* status, cudaStream_t stream) {
  using C = DkdvCfg<D, MODE, W>;
  auto kern = bwd_dkdv_kernel<D, BF16, MODE, KD, W>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const unsigned grid = static_cast<unsigned>((s.Nk + 127) / 128) * s.B * s.H;  // one CTA per KV tile
  return launch_dependent(kern, grid, C::kThreads, C::kSmemBytes, stream,
      tq, tk, tv, tdo, tdk, tdv, dk32, dv32, s.Dg, rowstats.stats, rowstats.tile_amax, dq_accum, s.N,
      s.Nk, s.B * s.H,
      s.H, heads_per_group(s), s.scale, s.scale * 1.4426950408889634f, status);
}

template <int D, bool BF16, int FORM, int KD = D>
cudaError_t launch_consume_t(const AttnShape& s, const void* scratch, const CUtensorMap& tb,
                             const CUtensorMap& tout, const F32Out& out32, const RowStats& rowstats, int* status,
                             cudaStream_t stream) {
  using C = ConsumeCfg<D>;
  auto kern = bwd_consume_kernel<D, BF16, FORM, KD>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const unsigned grid =
      static_cast<unsigned>(((FORM == 2 ? s.N : s.Nk) + 127) / 128) * s.B * s.H;  // one CTA per output tile
  return launch_dependent(kern, grid, C::kThreads, C::kSmemBytes, stream,
      static_cast<const uint4*>(scratch), tb, tout, out32, s.Dg, rowstats.tile_amax, s.N, s.Nk, s.B * s.H,
      s.H, heads_per_group(s), status);
}

template <bool BF16, int FORM, int KD>
cudaError_t launch_consume_pair_t(const AttnShape& s, const void* scratch, const CUtensorMap& tb,
                                  const CUtensorMap& tout, const F32Out& out32, const RowStats& rowstats,
                                  int* status, cudaStream_t stream) {
  using C = ConsumePairCfg;
  auto kern = bwd_consume_pair_kernel<BF16, FORM, KD>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const unsigned out_tiles = static_cast<unsigned>(((FORM == 2 ? s.N : s.Nk) + 127) / 128);
  return launch_dependent(kern, (out_tiles + 1) / 2 * s.B * s.H, C::kThreads, C::kSmemBytes, stream,
      static_cast<const uint4*>(scratch), tb, tout, out32, s.Dg, rowstats.tile_amax, s.N, s.Nk, s.B * s.H,
      s.H, heads_per_group(s), status);
}

template <int D, bool BF16, int KD = D, int W = 128>
cudaError_t launch_dq_t(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                        const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdq,
                        const F32Out& dq32, const RowStats& rowstats, int* status, cudaStream_t stream) {
  using C = DqCfg<D, W>;
  auto kern = bwd_dq_kernel<D, BF16, KD, W>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const unsigned grid = static_cast<unsigned>((s.N + 127) / 128) * s.B * s.H;  // one CTA per Q tile
  return launch_dependent(kern, grid, C::kThreads, C::kSmemBytes, stream,
      tq, tk, tv, tdo, tdq, dq32, s.Dg, rowstats.stats, rowstats.tile_amax, s.N, s.Nk, s.B * s.H, s.H,
      heads_per_group(s), s.scale, s.scale * 1.4426950408889634f, status);
}

}  // namespace

cudaError_t launch_bwd_dkdv(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                            const CUtensorMap& tv, const CUtensorMap& tdo,
                            const CUtensorMap& tdk, const CUtensorMap& tdv, const F32Out& dk32,
                            const F32Out& dv32, const RowStats& rowstats, float* dq_accum, int mode, int step_rows,
                            int* status, cudaStream_t stream) {
  // modes: 0 dK/dV only, 1 fused atomic dQ (dq_accum = fp32 accumulator), 2 spill dS tiles
  // (dq_accum = the 16-bit scratch tensor)
#define FA2_ARGS s, tq, tk, tv, tdo, tdk, tdv, dk32, dv32, rowstats, dq_accum, status, stream
  if (s.D == 128 && s.Dg <= kShortDim128 && mode == 2)
    return s.dtype ? launch_dkdv_t<128, true, 2, kShortDim128>(FA2_ARGS)
                   : launch_dkdv_t<128, false, 2, kShortDim128>(FA2_ARGS);
  if (s.D == 128 && s.Dg <= kShortDim128 && mode == 0)
    return s.dtype ? launch_dkdv_t<128, true, 0, kShortDim128>(FA2_ARGS)
                   : launch_dkdv_t<128, false, 0, kShortDim128>(FA2_ARGS);
  if (step_rows == 64) {
    if (s.D == 64 && mode == 1)
      return s.dtype ? launch_dkdv_t<64, true, 1, 64, 64>(FA2_ARGS) : launch_dkdv_t<64, false, 1, 64, 64>(FA2_ARGS);
    if (s.D == 64 && mode == 0)
      return s.dtype ? launch_dkdv_t<64, true, 0, 64, 64>(FA2_ARGS) : launch_dkdv_t<64, false, 0, 64, 64>(FA2_ARGS);
    if (s.D == 32 && mode == 1)
      return s.dtype ? launch_dkdv_t<32, true, 1, 32, 64>(FA2_ARGS) : launch_dkdv_t<32, false, 1, 32, 64>(FA2_ARGS);
    if (s.D == 32 && mode == 0)
      return s.dtype ? launch_dkdv_t<32, true, 0, 32, 64>(FA2_ARGS) : launch_dkdv_t<32, false, 0, 32, 64>(FA2_ARGS);
    return cudaErrorInvalidValue;
  }
#define FA2_CASE(DD)                                                                        \
  case DD:                                                                                  \
    if (mode == 1)                                                                          \
      return s.dtype ? launch_dkdv_t<DD, true, 1>(FA2_ARGS)                                 \
                     : launch_dkdv_t<DD, false, 1>(FA2_ARGS);                               \
    if (mode == 2)                                                                          \
      return s.dtype ? launch_dkdv_t<DD, true, 2>(FA2_ARGS)                                 \
                     : launch_dkdv_t<DD, false, 2>(FA2_ARGS);                               \
    return s.dtype ? launch_dkdv_t<DD, true, 0>(FA2_ARGS)                                   \
                   : launch_dkdv_t<DD, false, 0>(FA2_ARGS);
  switch (s.D) {
    FA2_CASE(32)
    FA2_CASE(64)
    FA2_CASE(128)
  }
#undef FA2_CASE
#undef FA2_ARGS
  return cudaErrorInvalidValue;
}

cudaError_t launch_bwd_dq(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                          const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdq,
                          const F32Out& dq32, const RowStats& rowstats, int step_rows, int* status,
                          cudaStream_t stream) {
#define FA2_ARGS s, tq, tk, tv, tdo, tdq, dq32, rowstats, status, stream
  if (s.D == 128 && s.Dg <= kShortDim128)
    return s.dtype ? launch_dq_t<128, true, kShortDim128>(FA2_ARGS)
                   : launch_dq_t<128, false, kShortDim128>(FA2_ARGS);
  if (step_rows == 64) {
    if (s.D == 64) return s.dtype ? launch_dq_t<64, true, 64, 64>(FA2_ARGS) : launch_dq_t<64, false, 64, 64>(FA2_ARGS);
    if (s.D == 32) return s.dtype ? launch_dq_t<32, true, 32, 64>(FA2_ARGS) : launch_dq_t<32, false, 32, 64>(FA2_ARGS);
    return cudaErrorInvalidValue;
  }
#define FA2_CASE(DD)                                                   \
  case DD:                                                             \
    return s.dtype ? launch_dq_t<DD, true>(FA2_ARGS)                   \
                   : launch_dq_t<DD, false>(FA2_ARGS);
  switch (s.D) {
    FA2_CASE(32)
    FA2_CASE(64)
    FA2_CASE(128)
  }
#undef FA2_CASE
#undef FA2_ARGS
  return cudaErrorInvalidValue;
}

cudaError_t launch_bwd_scores_wide(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                                   const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdv,
                                   const F32Out& dv32, const RowStats& rowstats, void* ds_scratch, int* status,
                                   cudaStream_t stream) {
#define FA2_ARGS s, tq, tk, tv, tdo, tdv, dv32, rowstats, ds_scratch, status, stream
  if (s.Dg <= kShortDim256)
    return s.dtype ? launch_scores_wide_t<true, 3>(FA2_ARGS) : launch_scores_wide_t<false, 3>(FA2_ARGS);
  return s.dtype ? launch_scores_wide_t<true, 4>(FA2_ARGS) : launch_scores_wide_t<false, 4>(FA2_ARGS);
#undef FA2_ARGS
}

cudaError_t launch_bwd_consume(const AttnShape& s, int form, const void* scratch,
                               const CUtensorMap& tb, const CUtensorMap& tout, const F32Out& out32,
                               const RowStats& rowstats, bool two_tiles, int* status, cudaStream_t stream) {
#define FA2_ARGS s, scratch, tb, tout, out32, rowstats, status, stream
#define FA2_CASE(DD)                                                      \
  case DD:                                                                \
    return s.dtype ? launch_consume_t<DD, true, 2>(FA2_ARGS)              \
                   : launch_consume_t<DD, false, 2>(FA2_ARGS);
#define FA2_WIDE(FORM, KD)                                                                        \
  (two_tiles ? (s.dtype ? launch_consume_pair_t<true, FORM, KD>(FA2_ARGS)                         \
                        : launch_consume_pair_t<false, FORM, KD>(FA2_ARGS))                       \
             : (s.dtype ? launch_consume_t<256, true, FORM, KD>(FA2_ARGS)                         \
                        : launch_consume_t<256, false, FORM, KD>(FA2_ARGS)))
  if (s.D == 256 && s.Dg <= kShortDim256) {
    if (form == 1) return FA2_WIDE(1, kShortDim256);
    if (form == 2) return FA2_WIDE(2, kShortDim256);
  } else if (s.D == 256) {
    if (form == 1) return FA2_WIDE(1, 256);
    if (form == 2) return FA2_WIDE(2, 256);
  }
#undef FA2_WIDE
  if (form != 2) return cudaErrorInvalidValue;
  if (s.D == 128 && s.Dg <= kShortDim128)
    return s.dtype ? launch_consume_t<128, true, 2, kShortDim128>(FA2_ARGS)
                   : launch_consume_t<128, false, 2, kShortDim128>(FA2_ARGS);
  switch (s.D) {
    FA2_CASE(32)
    FA2_CASE(64)
    FA2_CASE(128)
  }
#undef FA2_CASE
#undef FA2_ARGS
  return cudaErrorInvalidValue;
}

}  // namespace fa2
