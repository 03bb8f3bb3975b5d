// Tile geometry shared by the attention kernels, and the host-side launcher interface
// between the translation units of the library.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <utility>

namespace fa2 {

// A 128-row tile of a [.., N, D] tensor is staged in shared memory as D/CH "chunk tiles" of
// [128 rows][CH elements]; CH*2 bytes is the swizzle span (128 B for D >= 64, 64 B for D = 32).
// This is exactly what one TMA box of (CH, 128, 1) with the matching swizzle mode produces,
// and what the tensor-core shared-memory descriptors below describe.
template <int D>
struct Tile {
  static_assert(D == 32 || D == 64 || D == 128 || D == 256, "tile width must be 32, 64, 128 or 256");
  static constexpr int kRows = 128;
  static constexpr int kChunkElems = D >= 64 ? 64 : 32;
  static constexpr int kChunks = D / kChunkElems;
  static constexpr int kRowBytes = kChunkElems * 2;             // 128 or 64
  static constexpr int kChunkTileBytes = kRows * kRowBytes;     // 16384 or 8192
  static constexpr int kTileBytes = kChunks * kChunkTileBytes;  // 128 * D * 2
  static constexpr int kAtomBytes = 8 * kRowBytes;              // 8-row swizzle atom
  static constexpr uint32_t kSwizzleMode = kRowBytes == 128 ? 2u : 4u;
  static constexpr uint32_t kSwizzleMask = kRowBytes == 128 ? 7u : 3u;
  static constexpr int kKStepsPerChunk = kChunkElems / 16;  // MMAs (K = 16) per chunk tile
};

// Byte offset of the 16-byte piece `piece` of row `row` inside one chunk tile, after the
// hardware XOR swizzle (address bits [4,7) ^= bits [7,10), restricted to the swizzle span).
template <int D>
__host__ __device__ __forceinline__ uint32_t swizzled_offset(uint32_t row, uint32_t piece) {
  const uint32_t off = row * Tile<D>::kRowBytes + piece * 16u;
  return off ^ (((off >> 7) & Tile<D>::kSwizzleMask) << 4);
}

// Same for a [128 rows][64 elements] 16-bit tile with 128-byte rows, whatever D is (used
// for the score-gradient tile, whose row length is the tile width 128, not D).
__host__ __device__ __forceinline__ uint32_t swizzled_offset_128B(uint32_t row, uint32_t piece) {
  const uint32_t off = row * 128u + piece * 16u;
  return off ^ (((off >> 7) & 7u) << 4);
}

// ----------------------------------------------------------------------------------------
// Host launchers (one per kernel family), defined in the .cu files of this directory.
// Tensor maps describe [B, H, N, D] tensors with box (CH, 128, 64 or 32, 1, 1).
// ----------------------------------------------------------------------------------------
struct AttnShape {
  int B, H;
  int N;      // query rows (rows of q, o, dout, dq, lse)
  int D;      // head dim the kernels are instantiated for: 32, 64, 128 or 256
  int dtype;  // 0 = fp16, 1 = bf16
  float scale;
  int Dg;     // head dim of the tensors in memory (a multiple of 8, <= D); the columns
              // Dg..D-1 are zeros on TMA loads and dropped on TMA stores
  int Nk;     // key rows (rows of k, v, dk, dv), 1 <= Nk <= N; the causal mask is aligned at
              // the top left: query row i sees keys 0 .. min(i, Nk - 1)
};

// Element strides of one [B, H, N, D] tensor (the last dimension is contiguous).
struct Strides {
  long long b, h, n;
};

// An output written as fp32 straight from a kernel's accumulators (p == nullptr: the output is 16-bit
// and goes through its tensor map).  Strides in elements, base 32-byte aligned.
struct F32Out {
  float* p;
  Strides st;
};

// What the backward preprocess leaves for the backward kernels: the tile-blocked row statistics
// and, one word per 128-row tile, the largest |dout| of the tile (16-bit pattern, sign cleared),
// both indexed from the first (batch, head) problem of the launch.
struct RowStats {
  const float* stats;         // [B*H][T][2][128]
  const unsigned* tile_amax;  // [B*H][T]
};

// Smallest instantiated head dim that holds `d` columns.
inline int padded_head_dim(int d) { return d <= 32 ? 32 : (d <= 64 ? 64 : (d <= 128 ? 128 : 256)); }

// Rows of the tiles a backward kernel walks past its resident tile, one CTA per resident tile of the `rows` of a
// head: Q and dO tiles of the dK/dV kernel (its spill mode always takes 128), K and V tiles of the dQ kernel.
// Up to head dim 64 steps of 64 rows with two CTAs on an SM win once there are CTAs to pair: a CTA that has its SM
// to itself takes 1.2 to 1.5 times as long in them, and so does the longest CTA of a launch that is not
// many times longer, which is why the line rises with the tiles a head has.  Both give the same bits.
// Whole backward, fp16, head dim 64, microseconds in steps of 64 / 128 rows, recompute and atomic mode:
//     512 rows: 160 CTAs 24.3 / 23.6 and 24.9 / 24.1, 192 CTAs 25.3 / 26.6 and 26.9 / 26.9, 512 CTAs 43 / 57 and 45 / 52
//    2048 rows: 320 CTAs 69.4 / 68.9 and 62.9 / 61.4, 384 CTAs 73.7 / 79.3 and 65.8 / 69.9, 144 CTAs 67.6 / 46.5 and 49.6 / 43.4
//    8192 rows: 384 CTAs 271 / 229 and 211 / 202, 512 CTAs 301 / 309 and 249 / 260, 128 CTAs 217 / 146 and 155 / 127
//   32768 rows: 256 CTAs 872 / 552 and 680 / 461, 512 CTAs 1145 / 1141 and 935 / 963, 1024 CTAs 2191 / 2271 and 1843 / 1898
// (head dim 32, 8192 rows, 512 CTAs: 263 / 251 and 189 / 203).
inline int bwd_step_rows(const AttnShape& s, int rows, bool atomic, int num_sms) {
  const int tiles = (rows + 127) / 128;
  const int percent = tiles <= 4 ? 125 : (tiles <= 16 ? 240 : (atomic ? 330 : 360));  // CTAs a hundred SMs
  return s.D <= 64 && 100ll * tiles * s.B * s.H >= static_cast<long long>(percent) * num_sms ? 64 : 128;
}

// Rows of the KV tiles the forward kernel walks (its K and V tensor maps use boxes of this height): 64, with two
// CTAs on an SM, up to head dim 64 and 1024 rows.  The two forms round differently (other rescale points,
// other exponentials), so the rule looks at nothing but the head dim and the rows: O, and with it every
// gradient, keeps its bits however a batch is split.  Where the work fills the GPU 64 rows win up to about 4096
// rows at head dim 64 and everywhere at 32; where it does not they lose, the more the longer the rows.
// fp16, head dim 64, microseconds with 64 / 128 rows (single-tile items below where they are taken):
//     512 rows: 256 heads 27.9 / 34.4, 128: 18.5 / 18.4, 64: 13.5 / 11.7, 8: 12.3 / 12.2
//    1000 rows: 256 heads 68.3 / 85.4, 128: 35.9 / 43.6, 64: 26.1 / 24.2, 16: 19.5 / 18.2
//    2048 rows: 48 heads 53.2 / 49.0, 32: 50.7 (38.9) / 32.7, 8: 33.6 (29.9) / 27.2
//    4096 rows: 64 heads 203 / 210, 32: 104 / 100, 16: 91.6 (66.5) / 51.2, 4: 61.1 (54.7) / 48.2
//   16384 rows: 16 heads 766 / 721, 4: 337 (246) / 177;   32768 rows: 8 heads 1500 / 1385, 2: 669 (486) / 347
// (head dim 32: 4096 rows, 64 heads 172 / 187; 32768 rows, 8 heads 1199 / 1215).  Up to 1024 rows the loss
// with few heads stays at 2 us of a call that takes some 20 us on the host.
inline int fwd_kv_rows(const AttnShape& s) { return s.D <= 64 && s.N <= 1024 ? 64 : 128; }

// Q tiles of a work item of the 64-row form: two that share every K and V tile, or one where there are few, so that
// they spread over more CTAs and no CTA is left with a long pair.  Microseconds, one / two, head dim 64: 1000
// rows: 16 heads 19.5 / 21.5, 64: 26.1 / 29.8, 128: 47.7 / 35.9; 512 rows: 80 heads 13.7 / 17.9, 128: 18.8 / 18.5,
// 256: 34.7 / 27.9; 300 rows: 64 heads 10.3 / 10.2, 128: 15.1 / 12.9.  Same bits.
inline int fwd_tiles_per_item(const AttnShape& s, int num_sms) {
  const long long tiles = (s.N + 127) / 128;
  return 2 * tiles * s.B * s.H <= (tiles <= 3 ? 4 : 7) * static_cast<long long>(num_sms) ? 1 : 2;
}

// Order in which the causal kernels take their (head, tile) work items.  A tile's work shrinks
// with its rank (rank 0 is the tile that meets the most tiles of the other kind), so for an even
// finish the long items must start first; but the items of one head share its tensors through
// the L2 cache, so they must also run close together.  Heads are therefore taken in groups of
// `group` whose tensors fit a share of the L2 cache together, and inside a group every head's
// rank-0 item comes first, then every head's rank-1 item, and so on.  Against the plain
// head-by-head order this removes most of the causal tail (the last head's longest item no
// longer starts last): the fewer heads a launch has, the more it gains.
struct HeadTile {
  int bh;    // flattened (batch, head) index
  int rank;  // 0 = the heaviest tile of the head
};
__host__ __device__ __forceinline__ HeadTile grouped_order(long long id, int num_bh, int tiles,
                                                           int group) {
  const long long per_group = static_cast<long long>(group) * tiles;
  const int g0 = static_cast<int>(id / per_group) * group;
  const int n = num_bh - g0 < group ? num_bh - g0 : group;  // heads of this group
  const int local = static_cast<int>(id - (id / per_group) * per_group);
  return HeadTile{g0 + local % n, local / n};
}
// Heads per group: q, dout (or o) and k, v of the group's heads in 64 MiB of the 126 MiB L2.
inline int heads_per_group(const AttnShape& s) {
  const long long per_head = (2ll * s.N + 2ll * s.Nk) * s.D * 2;
  const long long g = (64ll << 20) / per_head;
  const long long bh = static_cast<long long>(s.B) * s.H;
  return static_cast<int>(g < 1 ? 1 : (g > bh ? bh : g));
}

// Per-launch context of the forward kernel.  It runs one or two CTAs per SM.  With more work items (Q tiles or pairs of
// them) than CTAs, these draw items from `work_counter` until none are left, so tensor memory is
// allocated once and no SM idles between items.  The counter is zero before the launch; a launch draws
// total_items + gridDim.x numbers in all, and whoever draws the last one puts the counter back to zero,
// so no memset sits between launches.
struct LaunchCtx {
  int* status;                 // device status word (bounded-wait failures)
  unsigned int* work_counter;  // device word, 0 at kernel start and again at kernel end
  int num_sms;
};

// Launches a kernel that may overlap the end of its predecessor on the stream (grid_wait_previous and
// grid_allow_next in ptx.cuh).  A successor without the attribute, a memset or an event still waits for the
// whole kernel.  Launch, set-up and the last wave of a kernel are what this covers; microseconds, plain
// launches against these: backward [4,16,2048,64] recompute 172 / 185 -> 167 / 171, atomic 173 -> 166,
// [8,16,1000,64] 113 -> 107, [8,12,4095,32] 757 -> 736, [32,20,1024,96] 782 -> 764, [2,16,8192,256] 3175
// -> 3065; forward [4,16,2048,64] 64.5 -> 59; [2,32,8192,128] unchanged.
template <typename... Params, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), unsigned grid, int threads, int smem_bytes,
                                    cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

cudaError_t launch_fwd(const AttnShape& s, int kv_rows, const CUtensorMap& tq, const CUtensorMap& tk,
                       const CUtensorMap& tv, const CUtensorMap& to, const F32Out& o32, float* lse,
                       const LaunchCtx& ctx, cudaStream_t stream);

// rowstats[bh][t][0][r] = -lse * log2(e) (-inf for padded rows), rowstats[bh][t][1][r] = -delta;
// behind the last tile, one 32-bit word per tile: the largest |dout| of the tile's rows as its
// 16-bit pattern with the sign cleared.  Tensors whose rows are not contiguous are read through `to` and `tdo`
// (boxes of 128 whole rows, 64 above head dim 128, no swizzle), which need not be valid otherwise.
cudaError_t launch_bwd_preprocess(const AttnShape& s, const CUtensorMap& to, const CUtensorMap& tdo,
                                  const void* o, const Strides& so, const void* dout, const Strides& sdo, const float* lse,
                                  float* rowstats, int* status, int num_sms,
                                  cudaStream_t stream);

// dK/dV per KV tile.  mode 1 also accumulates dQ into dq_accum with fp32 atomic adds
// (dq_accum layout: [bh][t][w = 4][k = D/4][lane = 32][4] floats, holding element
// (row 128*t + 32*w + lane, col 4*k + 0..3)); mode 2 also stores every 16-bit dS^T tile to the
// scratch tensor dq_accum then points to (32 KiB per (KV tile, Q tile) pair, pairs numbered
// per head KV tile by KV tile, see dstile_pairs), from which launch_bwd_consume (form 2) forms dQ.
cudaError_t launch_bwd_dkdv(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                            const CUtensorMap& tv, const CUtensorMap& tdo,
                            const CUtensorMap& tdk, const CUtensorMap& tdv, const F32Out& dk32,
                            const F32Out& dv32, const RowStats& rowstats, float* dq_accum, int mode, int step_rows,
                            int* status, cudaStream_t stream);

// Head dims above 128: dV per KV tile, and dS^T of every (KV tile, Q tile) pair as 16-bit piece-major tiles into a
// scratch tensor (pair numbering as in the spill mode); launch_bwd_consume forms 1 and 2 then give dK and dQ.
cudaError_t launch_bwd_scores_wide(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                                   const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdv,
                                   const F32Out& dv32, const RowStats& rowstats, void* ds_scratch, int* status,
                                   cudaStream_t stream);

// One output tile per CTA from spilled 16-bit score-gradient tiles, one product
// per tile pair in ascending order (deterministic):
//   form 2: dQ(qt) = sum_j dS(j, qt) K_j     (tb = K, tout = dQ)
//   form 1: dK(jt) = sum_i dS(jt, i)^T Q_i   (tb = Q, tout = dK)  head dim 256
// At head dim 256, with two_tiles, a CTA forms two adjacent output tiles (tb then has boxes of 64 rows).
cudaError_t launch_bwd_consume(const AttnShape& s, int form, const void* scratch,
                               const CUtensorMap& tb, const CUtensorMap& tout, const F32Out& out32,
                               const RowStats& rowstats, bool two_tiles, int* status, cudaStream_t stream);

// Whether the consumers of head dim 256 take two output tiles per CTA: when that still gives every SM a CTA.
// Below, fewer and longer CTAs leave SMs idle.  Whole bf16 backward, microseconds, one tile against two, head dim 256 and 192:
//     1024 rows: 128 pairs of tiles 85 / 88 and 87 / 90, 160: 118 / 109 and 123 / 113, 256: 160 / 151 and 170 / 157, 512: 292 / 275 and 288 / 274
//     2048 rows: 128 pairs 116 / 127 and 108 / 125, 160: 185 / 172 and 167 / 162, 256: 233 / 214 and 197 / 183, 320: 304 / 309 and 252 / 249
//     8192 rows: 128 pairs 350 / 414 and 298 / 337, 160: 595 / 578 and 527 / 479, 256: 661 / 620 and 553 / 518, 512: 1352 / 1253 and 1190 / 1072
inline bool consume_two_tiles(const AttnShape& s, int num_sms) {
  const long long tiles = (s.Nk + 127) / 128;
  return s.D == 256 && (tiles + 1) / 2 * s.B * s.H > num_sms;
}

// (KV tile, Q tile) pairs of one head: KV tile t < nktiles meets Q tiles t .. ntiles-1.
inline long long dstile_pairs(int N, int Nk) {
  const long long nt = (N + 127) / 128, nk = (Nk + 127) / 128;
  return nk * nt - nk * (nk - 1) / 2;
}

// dQ per Q tile, ascending KV order (deterministic path).
cudaError_t launch_bwd_dq(const AttnShape& s, const CUtensorMap& tq, const CUtensorMap& tk,
                          const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdq,
                          const F32Out& dq32, const RowStats& rowstats, int step_rows, int* status,
                          cudaStream_t stream);

// dq = convert(dq_accum) (non-deterministic path); into dq32 when that is given.
cudaError_t launch_dq_convert(const AttnShape& s, const float* dq_accum, void* dq,
                              const Strides& sdq, const F32Out& dq32, cudaStream_t stream);

// One CTA whose waits run into the time limit on purpose (nothing ever arrives); it must end
// by itself with the status word set.
cudaError_t launch_selftest_wait(int* status, cudaStream_t stream);

cudaError_t launch_selftest_mma(int form, const CUtensorMap& ta, const CUtensorMap& tb,
                                const void* a_raw, float* c, int D, int dtype, int* status,
                                cudaStream_t stream);

}  // namespace fa2
