// Causal attention forward for sm_100a.
//
// Replaces _forward_kernel (src/flash_attention_triton/_triton_kernels_v2.py:11-189 of the
// reference).  One CTA owns two adjacent 128-row Q tiles of one (batch, head) and walks the KV
// tiles 0..diagonal.  (What follows describes 128-row KV tiles, the last paragraph 64-row ones.)  Warp roles:
//   warps 0-3   softmax for Q tile 0   (thread = one score row = one tensor-memory lane)
//   warps 4-7   softmax for Q tile 1
//   warp  8     issues S = Q_i K_j^T          } one elected lane each; two warps so that neither
//   warp  10    issues O_i += P_i V_j         } MMA stream waits behind the other's barriers
//   warp  9     draws the work items; TMA producer: Q once an item, then a K ring and a V ring
//   warp  11    idle; warps 8-11 give registers to the softmax groups (setmaxnreg)
// (role numbers; hardware warps 0-3 take roles 8-11, see below)
//
// Tensor memory: ONE score buffer S shared by both Q tiles, a 16-bit probability buffer P_i per
// tile and an output accumulator O_i per tile.  A softmax group copies its score row into
// registers as soon as S is complete and hands the buffer back at once, so the next S product
// (for the other tile) runs while the group is still exponentiating; because P_i has its own
// columns, S_i(j+1) does not wait for O_i += P_i(j) V_j either.  Neither softmax group ever
// waits for its own MMAs in steady state: the tensor pipe sees four tile products per KV step
// back to back.
//
// The online softmax works in the exp2 domain with the scale folded in, and rescales O only
// when the running maximum has moved by more than kRescaleThreshold ("lazy rescale"); masking code runs on
// the diagonal tile only.  The exponentials go to the MUFU, although 2 x 128 x 128 of them a KV step cost as
// many cycles there (16 / clk / SM) as the four products: under load the power limit sets the clock, and a
// polynomial on the FMA pipe takes five times the instructions.  With 3 of 8 pairs in the polynomial against
// none, passes in a loop, microseconds: [2,32,8192,128] bf16 974 -> 921, [1,32,4096,128] 138 -> 129.5,
// [32,20,1024,96] fp16 223 -> 212, [2,16,8192,256] bf16 974 -> 926, [2,16,8192,64] fp16 373 -> 361.  At
// head dim 32, where the products are shortest, 3 of 8 pairs measure best, with 3 / 2 / none: [8,12,4095,32] fp16
// 258 / 259 / 267, [2,16,8192,32] 321 / 325 / 342, [1,2,32768,32] 343 / 350 / 384, [4,16,2048,32] 53.4 / 53.5 / 54.0.
//
// Head dims up to 64, rows up to fwd_kv_rows' line: the MMAs of a tile are short (512 cycles or less per 128 x 128 scores) and the
// softmax instruction stream is what takes the time; with two softmax warps per scheduler it issues
// in half of the cycles only, the rest is latency of dependent instructions.  So the KV tiles are
// 64 rows there: a thread holds 64 instead of 128 scores, 96 registers do instead of 208, 256
// columns of tensor memory instead of 512, and TWO CTAs run on an SM, four softmax warps per
// scheduler.  Measured against 128-row tiles and one CTA, fp16, head dim 64, microseconds:
// [1,256,1000,64] 85.4 -> 68.3, [1,128,1000,64] 43.6 -> 35.9, [1,256,512,64] 34.4 -> 27.9; where there are too
// few CTAs to pair, or the rows are long, 128-row tiles win (figures at fwd_kv_rows).
#include "common.cuh"
#include "mma_issue.cuh"
#include "ptx.cuh"

namespace fa2 {
namespace {

constexpr int kFwdThreads = 384;
constexpr float kLn2 = 0.6931471805599453f;

template <int D, int W>
struct FwdCfg {
  using T = Tile<D>;
  static constexpr int kW = W;  // rows of a KV tile = columns of a score tile
  static_assert(W == 128 || (W == 64 && D <= 64), "fwd_kv_rows");
  static constexpr int kPolyShare = kW == 128 && D == 32 ? 3 : 0;  // of every 8 column pairs, this many use ex2_poly2
  static constexpr int kCtasPerSm = kW == 64 ? 2 : 1;
  // O is rescaled when the running maximum has moved by more than this (log2 units).  A row's
  // largest P is exactly 1, without rounding error, when its maximum is fresh: 64-row tiles, whose
  // maxima settle later, use a lower threshold and none after their first tile, which keeps the
  // error of O below that of 128-row tiles (peaked softmax, fp16: 1.78e-4 against 1.84e-4).
  static constexpr float kRescaleThreshold = kW == 64 ? 4.0f : 8.0f;
  static constexpr int kKvBytes = T::kTileBytes / 128 * kW;
  // registers of a producer / softmax thread; the launch gives every thread
  // kLaunchRegs (the launch bounds' limit, rounded down to a multiple of 8)
  static constexpr int kLaunchRegs = 65536 / (kFwdThreads * kCtasPerSm) / 8 * 8;
  static constexpr int kProducerRegs = kW == 64 ? 48 : 72;
  static constexpr int kSoftmaxRegs = kW == 64 ? 96 : 216;
  static_assert(128 * kProducerRegs + 256 * kSoftmaxRegs <= kFwdThreads * kLaunchRegs,
                "setmaxnreg.inc waits for registers that setmaxnreg.dec has released");
  // At head dim 128 a third K stage measured the same as two; the output staging takes its place.
  static constexpr int kKStages = D == 128 ? 2 : 4;
  static constexpr int kVStages = kKStages;
  // O is staged in its own memory, 32 rows of one chunk for each softmax warp, so that the next item's Q can be
  // loaded under the epilogue; in the 64-row form, where the other CTA of the SM fills the gap, in the Q
  // tiles (with own memory the rings lose a stage: [8,16,1000,64] 35.6 -> 37.8 us).
  static constexpr bool kStageInQ = kW == 64;
  static constexpr int kStageBytes = 32 * T::kRowBytes;
  static constexpr int kOffQ = 0;
  static constexpr int kOffK = kOffQ + 2 * T::kTileBytes;
  static constexpr int kOffV = kOffK + kKStages * kKvBytes;
  static constexpr int kOffStage = kOffV + kVStages * kKvBytes;  // one piece for each softmax warp
  static constexpr int kOffBar = kOffStage + (kStageInQ ? 0 : 8 * kStageBytes);
  // barrier slots
  static constexpr int kBarItemFull = 0;   // 2: the work item in slot n % 2 may be read
  static constexpr int kBarItemEmpty = 2;  // 2: every role but the producer has read it (10 arrivals)
  static constexpr int kBarQFull = 4;
  static constexpr int kBarQEmpty = 5;     // the item's last score product, or its last store, has read the Q tiles
  static constexpr int kBarKFull = 6;
  static constexpr int kBarKEmpty = kBarKFull + kKStages;
  static constexpr int kBarVFull = kBarKEmpty + kKStages;
  static constexpr int kBarVEmpty = kBarVFull + kVStages;
  static constexpr int kBarSFull = kBarVEmpty + kVStages;  // 2: S holds tile i's scores
  static constexpr int kBarSFree = kBarSFull + 2;    // 2: group i has copied S out (4 arrivals)
  static constexpr int kBarPFull = kBarSFree + 2;    // 2: P_i written, O_i rescaled (4 arrivals)
  static constexpr int kBarPvDone = kBarPFull + 2;   // 2: O_i += P_i V completed
  static constexpr int kNumBars = kBarPvDone + 2;
  static constexpr int kOffItems = (kOffBar + kNumBars * 8 + 15) / 16 * 16;  // 2 x WorkItem
  static constexpr int kSmemBytes = kOffItems + 2 * 16 + 16;  // + tmem slot, abort flag, next item
  // tensor-memory columns
  static constexpr int kColS = 0;
  static constexpr int kColP = kW;      // P0, then P1 (kW / 2 columns of 16-bit pairs each)
  static constexpr int kColO = 2 * kW;  // O0, then O1 (D columns each)
  static constexpr int kTmemCols = 512 / kCtasPerSm;
  static_assert(kColO + 2 * D <= kTmemCols, "tensor memory of one CTA");
  static_assert(kCtasPerSm * (kSmemBytes + 1024) <= 228 * 1024, "shared memory of one SM");
};

// What the producer leaves in an item slot: one Q tile, or two adjacent ones, of one (batch, head).
struct WorkItem {
  int pair;  // -1: no more items
  int bh, h, b;
};

enum FwdSite {
  kSiteLoadK = 1,
  kSiteLoadV,
  kSiteMmaQ,
  kSiteMmaK,
  kSiteMmaV,
  kSiteMmaP,
  kSiteMmaSFree,
  kSiteSoftS,
  kSiteSoftPv,
  kSiteSoftO,
  kSiteAlign,
  kSiteItem,
  kSiteLoadQ
};

template <int D, bool BF16, int KD, int W>
__global__ void __launch_bounds__(kFwdThreads, FwdCfg<D == 256 ? 128 : D, W>::kCtasPerSm)
    fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
               const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap to,
               const __grid_constant__ F32Out o32, int cols, float* __restrict__ lse, int N, int Nk,
               int num_bh, int num_heads, int group, float scale_log2, int tiles_per_item, int* status,
               unsigned int* work_counter) {
  // Head dim 256 ("wide") runs on the staging and tensor-memory plan of head dim 128 with ONE
  // Q tile per work item: the two Q slots hold the two 128-column halves of that tile, K and V
  // tiles stream through their rings as half tiles, S = Q_lo K_lo^T + Q_hi K_hi^T accumulates
  // over two products and O_lo / O_hi take the places of O0 / O1.  Only softmax group 0 works.
  constexpr bool WIDE = D == 256;
  constexpr int DT = WIDE ? 128 : D;    // columns of one staged tile
  constexpr int HALVES = WIDE ? 2 : 1;  // staged tiles per 128 rows
  using C = FwdCfg<DT, W>;
  using T = Tile<DT>;
  constexpr int KT = WIDE ? DT : KD;  // columns of a staged tile that the products run over
  constexpr int KT1 = WIDE ? KD - DT : KD;                            // and of the second half
  constexpr int kChunks1 = WIDE ? KT1 / T::kChunkElems : T::kChunks;  // chunks staged of the second half
  extern __shared__ __align__(1024) uint8_t smem[];

  // Role index: hardware warps 0-3 take roles 8-11 (MMA, TMA, idle, idle) and hardware warps
  // 4-11 the softmax roles 0-7, so the latency-critical MMA / TMA warps have the lowest
  // hardware warp ids on their schedulers.  The shift is a multiple of 4, so role % 4 is
  // still the tensor-memory lane quarter the hardware warp may access.
  const int warp = ((threadIdx.x >> 5) + 8) % 12;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {  // swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0) atomicCAS(status, 0, 0x20000 | kSiteAlign);
    return;
  }
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::kOffItems + 2 * sizeof(WorkItem));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* next_slot = reinterpret_cast<volatile int*>(tmem_slot + 2);
  auto bar = [&](int i) { return smem_base + C::kOffBar + 8u * i; };

  const int ntiles = (N + 127) >> 7;
  const int nktiles = (Nk + W - 1) / W;  // KV tiles of W rows
  const int per_item = WIDE ? 1 : (W == 128 ? 2 : tiles_per_item);  // Q tiles of a work item
  const int npairs = per_item == 1 ? ntiles : (ntiles + 1) >> 1;    // work items per (batch, head)
  const int total_items = npairs * num_bh;
  // KV tiles of an item's Q tile i: those up to its diagonal, or to the last key (N = query rows, Nk <= N = key
  // rows); 0 for a second tile that does not exist
  auto second_tile = [&](const WorkItem& item) { return per_item == 2 && 2 * item.pair + 1 < ntiles; };
  auto kv_tiles = [&](const WorkItem& item, int i) {
    return i == 1 && !second_tile(item) ? 0 : min((per_item * item.pair + i + 1) * (128 / W), nktiles);
  };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(C::kBarItemFull + i), 1);
      mbar_init(bar(C::kBarItemEmpty + i), 10);
    }
    mbar_init(bar(C::kBarQFull), 1);
    mbar_init(bar(C::kBarQEmpty), C::kStageInQ ? 8 : 1);
    for (int i = 0; i < C::kKStages; ++i) {
      mbar_init(bar(C::kBarKFull + i), 1);
      mbar_init(bar(C::kBarKEmpty + i), 1);
    }
    for (int i = 0; i < C::kVStages; ++i) {
      mbar_init(bar(C::kBarVFull + i), 1);
      mbar_init(bar(C::kBarVEmpty + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(C::kBarSFull + i), 1);
      mbar_init(bar(C::kBarSFree + i), 4);
      mbar_init(bar(C::kBarPFull + i), 4);
      mbar_init(bar(C::kBarPvDone + i), 1);
    }
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == 8) {
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

  // One or two CTAs per SM.  A CTA draws its items from a global counter, heaviest first within a group of heads
  // (grouped_order), unless there is one for each CTA.  The first one is drawn too: with item blockIdx.x to start with,
  // a CTA that finds no SM at the launch, because another stream or a collective holds some, kept a heavy item
  // for the end.  Beside a kernel on 4 / 20 SMs, microseconds, item blockIdx.x first against drawn: [1,2,32768,128] 507 -> 391 /
  // 539 -> 387, [2,16,8192,64] 396 -> 341 / 433 -> 378, [4,16,2048,64] 75.8 -> 61.5 / 79.9 -> 65.5; alone 409 -> 411, 340 -> 343, 54.0 -> 54.5
  // in a loop (the draw's latency).
  // The roles run through the items without meeting: the producer draws the next item while the last tiles of the one before are in
  // flight, and loads its first K tile and, once the last score product has read Q, its Q tiles, so that
  // the next item's scores are formed while the softmax groups finish this one.  Every barrier keeps
  // its phase from item to item.  What bounds short rows is this boundary; with all roles meeting there it took
  // some 4 us an item (Q and K loads, first scores, epilogue, one after the other).  Microseconds before and after,
  // passes in a loop: [32,20,1024,96] fp16 246 -> 223, [4,16,2048,64] fp16 63.4 -> 56.1, [8,12,4095,32] fp16 282 ->
  // 258, [4,16,1000,64] bf16 25.7 -> 23.9, [2,32,8192,128] bf16 973 -> 974, [1,2,32768,128] 463 -> 471.
  //
  // Slot of the n-th item of this CTA, for every role but the producer; false: there is none, or the CTA gives up.
  // It votes.  The MMA warps' other waits do not (a vote in each: [8,16,1000,64] 35.4 -> 36.1 us, [4,16,2048,64] 54.5 -> 55.4), so
  // their lanes may leave one apart when the CTA gives up, some for the abort flag; they meet in a vote at the
  // end of the item, which every lane reaches.
  auto take_item = [&](int n, WorkItem& item) {
    if (!mbar_wait_warp(bar(C::kBarItemFull + (n & 1)), (n >> 1) & 1, w, kSiteItem)) return false;
    item = reinterpret_cast<const WorkItem*>(smem + C::kOffItems)[n & 1];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(C::kBarItemEmpty + (n & 1)));
    return item.pair >= 0;
  };

  if (warp >= 8) {
    reg_dec<C::kProducerRegs>();  // whole warpgroup (warps 8-11) gives registers to the softmax groups
    if (warp == 9) {
      // ---------------------------------------------------------------- TMA producer
      // (whole warp, converged; only the elected lane arms barriers and issues copies)
      const uint32_t elected = elect_one();
      if (elected) {
        prefetch_tensormap(&tq);
        prefetch_tensormap(&tk);
        prefetch_tensormap(&tv);
      }
      bool ok = true;
      int ks = 0, kph = 0, vs = 0, vph = 0;  // ring positions
      unsigned drawn = blockIdx.x;  // an item, or beyond total_items
      const bool draws = total_items > static_cast<int>(gridDim.x);
      auto draw = [&]() {
        if (lane == 0) drawn = draws ? atomicAdd(work_counter, 1u) : total_items;
      };
      auto drawn_item = [&]() {  // the number drawn, for the whole warp
        if (lane == 0) {
          if (draws && drawn == total_items + gridDim.x - 1u) atomicExch(work_counter, 0u);
          *next_slot = static_cast<int>(drawn);
        }
        __syncwarp();
        const int id = *next_slot;
        __syncwarp();
        return id;
      };
      if (draws) draw();
      for (int n = 0;; ++n) {
        const int id = drawn_item();
        WorkItem item{-1, 0, 0, 0};
        if (id < total_items) {
          const HeadTile ht = grouped_order(id, num_bh, npairs, group);
          // the last pair of Q tiles meets the most KV tiles
          item = WorkItem{npairs - 1 - ht.rank, ht.bh, ht.bh % num_heads, ht.bh / num_heads};
        }
        if (ok) ok = mbar_wait_warp(bar(C::kBarItemEmpty + (n & 1)), ((n >> 1) & 1) ^ 1, w, kSiteItem);
        if (ok && lane == 0) {
          reinterpret_cast<WorkItem*>(smem + C::kOffItems)[n & 1] = item;
          mbar_arrive(bar(C::kBarItemFull + (n & 1)));
        }
        if (item.pair < 0) break;
        const HeadCoord hc{item.h, item.b};
        const int nkv = max(kv_tiles(item, 0), kv_tiles(item, 1));
        const int qt0 = per_item * item.pair;
        // K runs one KV tile ahead of V: S(j+1) is issued during KV step j.  Ring entries are
        // staged tiles: entry t holds columns (t % HALVES) * 128 .. of KV tile t / HALVES.
        const int nsub = nkv * HALVES;
        bool asked = false;  // the next item's number has been drawn
        for (int t = 0; ok && t < nsub + HALVES; ++t) {
          if (t < nsub) {
            if (!(ok = mbar_wait_warp(bar(C::kBarKEmpty + ks), kph ^ 1, w, kSiteLoadK))) break;
            if (elected) {
              const int chunks = t % HALVES ? kChunks1 : T::kChunks;
              mbar_arrive_expect_tx(bar(C::kBarKFull + ks), C::kKvBytes / T::kChunks * chunks);
#pragma unroll
              for (int ch = 0; ch < T::kChunks; ++ch)
                if (ch < chunks) tma_load_4d(smem_base + C::kOffK + ks * C::kKvBytes + ch * (C::kKvBytes / T::kChunks), &tk,
                            (t % HALVES) * 128 + ch * T::kChunkElems, (t / HALVES) * W, hc,
                            bar(C::kBarKFull + ks));
            }
            if (++ks == C::kKStages) ks = 0, kph ^= 1;
          }
          if (t == 0) {
            if (!(ok = mbar_wait_warp(bar(C::kBarQEmpty), (n & 1) ^ 1, w, kSiteLoadQ))) break;
            if (elected) {
              const int nslots = (WIDE || second_tile(item)) ? 2 : 1;
              mbar_arrive_expect_tx(bar(C::kBarQFull),
                                    WIDE ? T::kTileBytes + kChunks1 * T::kChunkTileBytes : nslots * T::kTileBytes);
              for (int i = 0; i < nslots; ++i)
                for (int ch = 0; ch < (WIDE && i ? kChunks1 : T::kChunks); ++ch)
                  tma_load_4d(smem_base + C::kOffQ + i * T::kTileBytes + ch * T::kChunkTileBytes, &tq,
                              (WIDE ? i * 128 : 0) + ch * T::kChunkElems, (WIDE ? qt0 : qt0 + i) * 128, hc,
                              bar(C::kBarQFull));
            }
          }
          if (t >= HALVES) {
            const int tv_ = t - HALVES;
            // the number of the next item is on its way while the last V tile waits for its stage
            if (tv_ == nsub - 1) {
              asked = true;
              draw();
            }
            if (!(ok = mbar_wait_warp(bar(C::kBarVEmpty + vs), vph ^ 1, w, kSiteLoadV))) break;
            if (elected) {
              const int chunks = tv_ % HALVES ? kChunks1 : T::kChunks;
              mbar_arrive_expect_tx(bar(C::kBarVFull + vs), C::kKvBytes / T::kChunks * chunks);
#pragma unroll
              for (int ch = 0; ch < T::kChunks; ++ch)
                if (ch < chunks) tma_load_4d(smem_base + C::kOffV + vs * C::kKvBytes + ch * (C::kKvBytes / T::kChunks), &tv,
                            (tv_ % HALVES) * 128 + ch * T::kChunkElems, (tv_ / HALVES) * W, hc,
                            bar(C::kBarVFull + vs));
            }
            if (++vs == C::kVStages) vs = 0, vph ^= 1;
            if (tv_ == nsub - 1) break;
          }
        }
        if (!asked) draw();  // a CTA that gives up goes on drawing, once an item, so that the counter is left at zero
      }
    } else if (warp == 8) {
      // ---------------------------------------------------------------- S = Q_i K_j^T issuer
      // Whole warp, converged; only the elected lane issues MMAs and commits.  The score
      // products and the P V products are issued by two different warps (this one and warp
      // 10): they touch disjoint tensor-memory columns and are ordered against each other
      // only through the softmax groups, so neither stream waits behind the other's barriers.
      // Order: S0(0) S1(0) S0(1) S1(1) ...; each product waits until the previous one has
      // been copied out of the single score buffer.  Releases are committed before the product's own
      // barrier, so that nothing is on its way to a barrier when the last item's outputs have been formed.
      const uint32_t elected = elect_one();
      auto commit = [&](int b) {
        if (elected) mma_commit(bar(b));
      };
      bool ok = true;
      int ks = 0, kph = 0;           // K ring position
      int prev_i = -1, prev_ph = 0;  // group and phase of the previous score product
      int count[2] = {0, 0};         // score products of either group so far
      auto release_k = [&]() {
        commit(C::kBarKEmpty + ks);
        if (++ks == C::kKStages) ks = 0, kph ^= 1;
      };
      WorkItem item;
      for (int n = 0; ok && take_item(n, item); ++n) {
        const int n0 = kv_tiles(item, 0), n1 = kv_tiles(item, 1), nkv = max(n0, n1);
        ok = mbar_wait(bar(C::kBarQFull), n & 1, w, kSiteMmaQ);
        for (int j = 0; ok && j < nkv; ++j) {
          if constexpr (!WIDE) {
            if (!(ok = mbar_wait(bar(C::kBarKFull + ks), kph, w, kSiteMmaK))) break;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (j >= (i == 0 ? n0 : n1)) continue;
            if (prev_i >= 0) {
              if (!(ok = mbar_wait(bar(C::kBarSFree + prev_i), prev_ph, w, kSiteMmaSFree))) break;
              tc_fence_after();
            }
            const bool last_of_tile = i == 1 || n1 == 0;
            if constexpr (WIDE) {
              // S = Q_lo K_lo^T + Q_hi K_hi^T: the Q slots hold the halves, K arrives half by half
              for (int half = 0; ok && half < 2; ++half) {
                if (!(ok = mbar_wait(bar(C::kBarKFull + ks), kph, w, kSiteMmaK))) break;
                const uint32_t qa = smem_base + C::kOffQ + half * T::kTileBytes, ka = smem_base + C::kOffK + ks * C::kKvBytes;
                if (KT1 == KT || half == 0)
                  issue_rows_x_rows<DT, BF16, W, KT>(elected, tmem_base + C::kColS, qa, ka, half);
                else
                  issue_rows_x_rows<DT, BF16, W, KT1>(elected, tmem_base + C::kColS, qa, ka, 1u);
                release_k();
              }
              if (!ok) break;
            } else {
              issue_rows_x_rows<DT, BF16, W, KT>(elected, tmem_base + C::kColS,
                                          smem_base + C::kOffQ + i * T::kTileBytes,
                                          smem_base + C::kOffK + ks * C::kKvBytes);
              if (last_of_tile) release_k();  // both products that read K_j issued
            }
            if (!C::kStageInQ && last_of_tile && j == nkv - 1) commit(C::kBarQEmpty);
            commit(C::kBarSFull + i);
            prev_i = i;
            prev_ph = count[i]++ & 1;
          }
        }
        ok = __all_sync(0xffffffffu, ok);  // see take_item
      }
    } else if (warp == 10) {
      // ---------------------------------------------------------------- O_i += P_i V_j issuer
      const uint32_t elected = elect_one();
      auto commit = [&](int b) {
        if (elected) mma_commit(bar(b));
      };
      bool ok = true;
      int vs = 0, vph = 0;    // V ring position
      int count[2] = {0, 0};  // products of either group so far
      auto release_v = [&]() {
        commit(C::kBarVEmpty + vs);
        if (++vs == C::kVStages) vs = 0, vph ^= 1;
      };
      WorkItem item;
      for (int n = 0; ok && take_item(n, item); ++n) {
        const int n0 = kv_tiles(item, 0), n1 = kv_tiles(item, 1), nkv = max(n0, n1);
        for (int j = 0; ok && j < nkv; ++j) {
          if constexpr (!WIDE) {
            if (!(ok = mbar_wait(bar(C::kBarVFull + vs), vph, w, kSiteMmaV))) break;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (j >= (i == 0 ? n0 : n1)) continue;
            if (!(ok = mbar_wait(bar(C::kBarPFull + i), count[i]++ & 1, w, kSiteMmaP))) break;
            tc_fence_after();
            if constexpr (WIDE) {
              // O_lo += P V_lo, O_hi += P V_hi: the O0 / O1 columns hold the two halves of O
              for (int half = 0; ok && half < 2; ++half) {
                if (!(ok = mbar_wait(bar(C::kBarVFull + vs), vph, w, kSiteMmaV))) break;
                const uint32_t o = tmem_base + C::kColO + half * DT, va = smem_base + C::kOffV + vs * C::kKvBytes;
                if (KT1 == KT || half == 0)
                  issue_tmem_x_tile<DT, BF16, W, KT>(elected, o, tmem_base + C::kColP, W / 4, va, j > 0);
                else
                  issue_tmem_x_tile<DT, BF16, W, KT1>(elected, o, tmem_base + C::kColP, W / 4, va, j > 0);
                release_v();
              }
              if (!ok) break;
            } else {
              issue_tmem_x_tile<DT, BF16, W, KT>(elected, tmem_base + C::kColO + i * DT,
                                          tmem_base + C::kColP + i * (W / 2), W / 4,
                                          smem_base + C::kOffV + vs * C::kKvBytes, j > 0);
              if (i == 1 || n1 == 0) release_v();
            }
            commit(C::kBarPvDone + i);
          }
        }
        ok = __all_sync(0xffffffffu, ok);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax groups
    reg_inc<C::kSoftmaxRegs>();
    const int wg = warp >> 2;
    const int r = (warp & 3) * 32 + lane;  // row inside the Q tile = tensor-memory lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem_base + lane_base + C::kColS;
    const uint32_t tP = tmem_base + lane_base + C::kColP + wg * (W / 2);
    const uint32_t tO = tmem_base + lane_base + C::kColO + wg * DT;  // wide: 256 columns, wg 0 only
    bool ok = true;
    int done = 0;  // KV tiles of this group's earlier items
    WorkItem item;
    for (int n = 0; ok && take_item(n, item); ++n) {
    const HeadCoord hc{item.h, item.b};
    const int qt = per_item * item.pair + wg;
    const int nj = kv_tiles(item, wg);
    float m_run = -INFINITY, l_run = 0.f;
    for (int j = 0; j < nj; ++j) {
      const int ph = (done + j) & 1;  // of this tile on the group's barriers
      if (!(ok = mbar_wait_warp(bar(C::kBarSFull + wg), ph, w, kSiteSoftS))) break;
      tc_fence_after();
      uint32_t sr[W];
#pragma unroll
      for (int c = 0; c < W; c += 32) tmem_ld_x32(tS + c, sr + c);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarSFree + wg));  // S may be overwritten now
      float* s = reinterpret_cast<float*>(sr);
      if (j * W + W > qt * 128 || j * W + W > Nk) {
        // diagonal tiles: keep col <= row; last KV tile: drop the columns beyond the last key
        const int last = min(qt * 128 + r, Nk - 1) - j * W;
#pragma unroll
        for (int c = 0; c < W; ++c) s[c] = (c <= last) ? s[c] : -INFINITY;
      }
      float mx[W / 32];
#pragma unroll
      for (int q4 = 0; q4 < W / 32; ++q4) {
        mx[q4] = max3(s[32 * q4], s[32 * q4 + 1], s[32 * q4 + 2]);
#pragma unroll
        for (int c = 3; c < 31; c += 2) mx[q4] = max3(mx[q4], s[32 * q4 + c], s[32 * q4 + c + 1]);
        mx[q4] = fmaxf(mx[q4], s[32 * q4 + 31]);
      }
      float m_new = max3(m_run, mx[0], mx[1]);
      if constexpr (W == 128) m_new = fmaxf(m_new, fmaxf(mx[2], mx[3]));
      const float threshold = W == 128 ? C::kRescaleThreshold : (j == 1 ? 0.f : C::kRescaleThreshold);
      const bool need = (m_new - m_run) * scale_log2 > threshold;
      bool pv_waited = false;
      if (__any_sync(0xffffffffu, need)) {
        // A neighbour's rescale must not touch a row without a finite score so far: -inf - -inf is no factor.
        const float alpha = m_new == -INFINITY ? 1.0f : ex2((m_run - m_new) * scale_log2);
        l_run *= alpha;
        m_run = m_new;
        if (j > 0) {
          // O_i must be at rest: wait for O_i += P_i(j-1) V_(j-1)
          if (!(ok = mbar_wait_warp(bar(C::kBarPvDone + wg), ph ^ 1, w, kSiteSoftPv))) break;
          tc_fence_after();
          pv_waited = true;
          constexpr int kStep = W == 64 ? 16 : 32;  // the score row stays in registers meanwhile
#pragma unroll
          for (int c0 = 0; c0 < KD; c0 += kStep) {
            uint32_t orr[kStep];
            if constexpr (kStep == 16) tmem_ld_x16(tO + c0, orr); else tmem_ld_x32(tO + c0, orr);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < kStep; ++c) orr[c] = __float_as_uint(__uint_as_float(orr[c]) * alpha);
            if constexpr (kStep == 16) tmem_st_x16(tO + c0, orr); else tmem_st_x32(tO + c0, orr);
          }
        }
      }
      // p = 2^(s*c - m*c) with packed fp32x2 FMAs; row sum in four independent packed chains.
      const float2 sc2 = make_float2(scale_log2, scale_log2);
      // A row whose scores so far are all -inf (infinite inputs, or finite ones whose product overflows) has
      // weights 0 (2^-126 from the polynomial) and not -inf + inf; its first finite score rescales them away.
      const float neg_m = m_run == -INFINITY ? 0.f : -m_run * scale_log2;
      const float2 nm2 = make_float2(neg_m, neg_m);
      float2 acc[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      uint32_t pk[W / 2];
#pragma unroll
      for (int c = 0; c < W / 2; ++c) {
        float2 t = __ffma2_rn(make_float2(s[2 * c], s[2 * c + 1]), sc2, nm2);
        if ((c & 7) < C::kPolyShare) {
          t = ex2_poly2(t);
        } else {
          t.x = ex2(t.x);
          t.y = ex2(t.y);
        }
        acc[c & 3] = __fadd2_rn(acc[c & 3], t);
        pk[c] = pack2<kInterBF16<BF16>>(t.x, t.y);
      }
      if (j > 0 && !pv_waited) {
        // P_i still feeds O_i += P_i(j-1) V_(j-1) until that product has completed
        if (!(ok = mbar_wait_warp(bar(C::kBarPvDone + wg), ph ^ 1, w, kSiteSoftPv))) break;
      }
#pragma unroll
      for (int c = 0; c < W / 2; c += 32) tmem_st_x32(tP + c, pk + c);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(C::kBarPFull + wg));
      const float2 a01 = __fadd2_rn(acc[0], acc[1]), a23 = __fadd2_rn(acc[2], acc[3]);
      l_run += (a01.x + a01.y) + (a23.x + a23.y);
    }
    done += nj;
    if (ok && nj > 0 && (ok = mbar_wait_warp(bar(C::kBarPvDone + wg), (done - 1) & 1, w, kSiteSoftO))) {
      tc_fence_after();
      // a row without any finite score has no softmax, whatever weights it was left with
      const float inv_l = m_run == -INFINITY ? __uint_as_float(0x7fffffffu) : 1.0f / l_run;
      // Each warp stages its own 32 rows, chunk by chunk, in the swizzled layout the output tensor map
      // expects, and stores them while the other roles are at the next item.
      const int row = qt * 128 + r, row0 = qt * 128 + (warp & 3) * 32;
      float* const dst32 =
          o32.p != nullptr && row < N ? o32.p + hc.b * o32.st.b + hc.h * o32.st.h + row * o32.st.n : nullptr;
#pragma unroll
      for (int c0 = 0; c0 < KD; c0 += 32) {
        uint32_t orr[32];
        tmem_ld_x32(tO + c0, orr);
        tmem_wait_ld();
        const int piece0 = (c0 % T::kChunkElems) / 8;
        uint8_t* const sO = C::kStageInQ ? smem + C::kOffQ + wg * T::kTileBytes + (warp & 3) * C::kStageBytes
                                         : smem + C::kOffStage + warp * C::kStageBytes;
        if (!C::kStageInQ && piece0 == 0) {
          // the staging piece may be refilled once the store before has READ it; the write itself
          // completes on its own before the grid does
          if (lane == 0) tma_store_wait_read();
          __syncwarp();
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          uint4 val;
          val.x = pack2<BF16>(__uint_as_float(orr[8 * p + 0]) * inv_l,
                              __uint_as_float(orr[8 * p + 1]) * inv_l);
          val.y = pack2<BF16>(__uint_as_float(orr[8 * p + 2]) * inv_l,
                              __uint_as_float(orr[8 * p + 3]) * inv_l);
          val.z = pack2<BF16>(__uint_as_float(orr[8 * p + 4]) * inv_l,
                              __uint_as_float(orr[8 * p + 5]) * inv_l);
          val.w = pack2<BF16>(__uint_as_float(orr[8 * p + 6]) * inv_l,
                              __uint_as_float(orr[8 * p + 7]) * inv_l);
          *reinterpret_cast<uint4*>(sO + swizzled_offset<DT>(lane, piece0 + p)) = val;
          // the unrounded row as well, for fp32 callers (see store_rows_f32 in bwd_roles.cuh)
          if (dst32 != nullptr && c0 + 8 * p < cols) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = __uint_as_float(orr[8 * p + i]) * inv_l;
            st_global_8(dst32 + c0 + 8 * p, x);
          }
        }
        if ((c0 + 32) % T::kChunkElems == 0 || c0 + 32 == KD) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && row0 < N) {
            tma_store_4d(&to, c0 / T::kChunkElems * T::kChunkElems, row0, hc, smem_u32(sO));
            tma_store_commit();
          }
        }
      }
      tc_fence_before();  // O_i is overwritten by the next item's first product, which this group's P lets in
      if (row < N)
        lse[static_cast<size_t>(item.bh) * N + row] = (m_run * scale_log2 + lg2(l_run)) * kLn2;
    }
    if constexpr (C::kStageInQ) {
      // A group without a tile has waited for nothing yet: its arrival must not count for the item before.
      if (ok && nj == 0) ok = mbar_wait_warp(bar(C::kBarQFull), n & 1, w, kSiteSoftO);
      if (lane == 0) tma_store_wait_read(), mbar_arrive(bar(C::kBarQEmpty));
    }
    }  // items
    if (lane == 0) tma_store_wait_read();
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int D, bool BF16, int KD = D, int W = 128>
cudaError_t launch_fwd_t(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                         const CUtensorMap& tv, const CUtensorMap& to, const F32Out& o32, float* lse,
                         const LaunchCtx& ctx, cudaStream_t stream) {
  using C = FwdCfg<D == 256 ? 128 : D, W>;  // head dim 256 runs on the plan of head dim 128
  auto kern = fwd_kernel<D, BF16, KD, W>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const int ntiles = (s.N + 127) / 128;
  const int tiles_per_item = D == 256 ? 1 : (W == 128 ? 2 : fwd_tiles_per_item(s, ctx.num_sms));
  const long long items = static_cast<long long>((ntiles + tiles_per_item - 1) / tiles_per_item) * s.B * s.H;
  const long long slots = static_cast<long long>(ctx.num_sms) * C::kCtasPerSm;
  const unsigned grid = static_cast<unsigned>(items < slots ? items : slots);
  const float scale_log2 = s.scale * 1.4426950408889634f;
  return launch_dependent(kern, grid, kFwdThreads, C::kSmemBytes, stream,
      tq, tk, tv, to, o32, s.Dg, lse, s.N, s.Nk, s.B * s.H, s.H, heads_per_group(s), scale_log2,
      tiles_per_item, ctx.status, ctx.work_counter);
}

}  // namespace

cudaError_t launch_fwd(const AttnShape& s, int kv_rows, const CUtensorMap& tq, const CUtensorMap& tk,
                       const CUtensorMap& tv, const CUtensorMap& to, const F32Out& o32, float* lse,
                       const LaunchCtx& ctx, cudaStream_t stream) {
  if (kv_rows == 64)
    return s.D == 64 ? (s.dtype ? launch_fwd_t<64, true, 64, 64>(s, tq, tk, tv, to, o32, lse, ctx, stream)
                                : launch_fwd_t<64, false, 64, 64>(s, tq, tk, tv, to, o32, lse, ctx, stream))
                     : (s.dtype ? launch_fwd_t<32, true, 32, 64>(s, tq, tk, tv, to, o32, lse, ctx, stream)
                                : launch_fwd_t<32, false, 32, 64>(s, tq, tk, tv, to, o32, lse, ctx, stream));
#define FA2_CASE(DD)                                                                 \
  case DD:                                                                           \
    return s.dtype ? launch_fwd_t<DD, true>(s, tq, tk, tv, to, o32, lse, ctx, stream)     \
                   : launch_fwd_t<DD, false>(s, tq, tk, tv, to, o32, lse, ctx, stream);
  if (s.D == 128 && s.Dg <= kShortDim128)
    return s.dtype ? launch_fwd_t<128, true, kShortDim128>(s, tq, tk, tv, to, o32, lse, ctx, stream)
                   : launch_fwd_t<128, false, kShortDim128>(s, tq, tk, tv, to, o32, lse, ctx, stream);
  if (s.D == 256 && s.Dg <= kShortDim256)
    return s.dtype ? launch_fwd_t<256, true, kShortDim256>(s, tq, tk, tv, to, o32, lse, ctx, stream)
                   : launch_fwd_t<256, false, kShortDim256>(s, tq, tk, tv, to, o32, lse, ctx, stream);
  switch (s.D) {
    FA2_CASE(32)
    FA2_CASE(64)
    FA2_CASE(128)
    FA2_CASE(256)
  }
#undef FA2_CASE
  return cudaErrorInvalidValue;
}

}  // namespace fa2
