// Bandwidth-bound helpers of the backward pass.
//
//   bwd_preprocess_ring_kernel  delta[row] = sum_d float(o[row,d]) * float(dout[row,d])
//       replaces _backward_preprocess_do_o_dot (_triton_kernels_v2.py:532-608 of the
//       reference).  Algorithmic traffic per row: 2 * D * 2 bytes read + 4 bytes (lse) read +
//       8 bytes written.
//   dq_convert_kernel      dq = 16-bit(dq_accum), the single fp32 -> 16-bit rounding the
//       reference performs with dq.copy_(dq_accum) (flash_attention_2.py:277).
#include "common.cuh"
#include "ptx.cuh"

namespace fa2 {
namespace {

template <bool BF16>
__device__ __forceinline__ float dot8(const uint4& a, const uint4& b) {
  const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
  const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 fa, fb;
    if constexpr (BF16) {
      fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i]));
      fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bw[i]));
    } else {
      fa = __half22float2(*reinterpret_cast<const __half2*>(&aw[i]));
      fb = __half22float2(*reinterpret_cast<const __half2*>(&bw[i]));
    }
    acc = fmaf(fa.x, fb.x, acc);
    acc = fmaf(fa.y, fb.y, acc);
  }
  return acc;
}

constexpr float kLog2e = 1.4426950408889634f;

// ----------------------------------------------------------------------------------------
// The preprocess: a persistent kernel fed by the copy engine.
//
// One CTA per SM walks the 128-row tiles blockIdx.x, blockIdx.x + gridDim.x, ...  A producer warp
// keeps a ring of shared-memory stages full (one stage = the o rows and the dout rows of one tile, or of half a tile
// at head dims above 128; an untiled bulk copy per tensor when its rows are contiguous in memory, else a tiled one
// through its tensor map), so the bytes in flight per SM stay near the ring size (128 - 192 KiB) whatever
// the eight consumer warps are doing; a block per tile has nothing in flight while
// it reduces and stores, and reaches less than half of the HBM rate ([2,16,8192,256] bf16, inside a step: 125 us, now 87).
// A group of D/8 adjacent lanes owns a row: each lane multiplies one 16-byte piece of o and of dout, and the group
// reduces with shuffles in a fixed order (deterministic).  The lanes beyond the d8 pieces of a row contribute zeros.
// Consumers free the stage once every piece has been used, and hand the tile's 256 results to the next iteration,
// which stores them with one coalesced 1 KiB write.  lse of the next tile is fetched one
// iteration ahead.  Rows in shared memory are packed at their true width (d8 pieces).  Rows beyond N are written
// too: -lse2 = -inf makes every probability of a padded row exactly 0 downstream.  Both vectors are stored NEGATED so
// that the consumers can use them as FMA / ADD addends directly.  The largest |dout| of a tile goes, as the
// 16-bit pattern with the sign cleared, to tile_amax[tile] (see head_dscale in bwd_roles.cuh).
// Rows apart from each other (dout as a projection behind it works on it, [B,N,H,d]) came in one bulk copy each,
// 64 to 256 bytes at a time; as tiled copies they cost what contiguous rows do.  Microseconds, copies of a row /
// tiled / contiguous rows: [8,16,1000,64] 37 / 13 / 12, [8,12,4095,32] 96 / 21 / 21, [32,20,1024,96] 162 / 49 / 49,
// [2,32,8192,128] 135 / 50 / 49.
// ----------------------------------------------------------------------------------------
template <int D>
struct PreRing {
  static constexpr int kRows = D == 256 ? 64 : 128;   // of a stage
  static constexpr int kParts = 128 / kRows;          // stages of a tile
  static constexpr int kPartBytes = kRows * D * 2;    // one tensor's rows at the padded width
  static constexpr int kStageBytes = 2 * kPartBytes;  // o, then dout
  static constexpr int kStages = D >= 128 ? 3 : (D == 64 ? 6 : 8);
  static constexpr int kConsumers = 256;
  static constexpr int kThreads = kConsumers + 32;
  // after the stages: full / empty barriers, two result buffers of 256 floats, two of 8 maxima
  static constexpr int kOffBars = kStages * kStageBytes;
  static constexpr int kOffStat = kOffBars + 16 * kStages;
  static constexpr int kOffMax = kOffStat + 2 * 256 * 4;
  static constexpr int kOffAbort = kOffMax + 2 * 8 * 4;
  static constexpr int kSmemBytes = kOffAbort + 16;
};

enum PreSite { kPSiteProducer = 64, kPSiteConsumer };

// All consumer threads learn whether every one of them got its stage (they leave together).
__device__ __forceinline__ bool consumers_all(bool ok, int nthreads) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "barrier.cta.red.and.pred p, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(ok)), "r"(nthreads)
      : "memory");
  return r != 0;
}

template <int D, bool BF16>
__global__ void __launch_bounds__(PreRing<D>::kThreads, 1)
    bwd_preprocess_ring_kernel(const __grid_constant__ CUtensorMap to, const __grid_constant__ CUtensorMap tdo,
                               const uint4* o, const uint4* dout, const float* lse, float* __restrict__ rowstats,
                               unsigned* __restrict__ tile_amax, int N, int ntiles,
                               long long tiles, int d8, int H, Strides so, Strides sdo,
                               int* status) {
  using R = PreRing<D>;
  constexpr int kLanesPerRow = D / 8;
  constexpr int kRowsPerPass = R::kConsumers / kLanesPerRow;  // 64, 32, 16 or 8
  constexpr int kPasses = R::kRows / kRowsPerPass;            // of a stage: 2, 4 or 8
  constexpr int kTilePasses = R::kParts * kPasses;
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t base = smem_u32(smem);
  auto full = [&](int s) { return base + R::kOffBars + 16u * s; };
  auto empty = [&](int s) { return base + R::kOffBars + 16u * s + 8u; };
  float* stat = reinterpret_cast<float*>(smem + R::kOffStat);
  unsigned* wmax = reinterpret_cast<unsigned*>(smem + R::kOffMax);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + R::kOffAbort);
  const WaitCtx w{abort_flag, status};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < R::kStages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), R::kConsumers / 32);
    }
    fence_mbar_init();
  }
  __syncthreads();
  grid_wait_previous();
  grid_allow_next();
  const uint32_t row_bytes = static_cast<uint32_t>(d8) * 16u;

  if (warp == R::kConsumers / 32) {
    // ---------------- producer warp ----------------
    int s = 0, ph = 0;
    bool ok = true;
    for (long long tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
      const long long bh = tile / ntiles;
      const int t = static_cast<int>(tile - bh * ntiles);
      const long long bb = bh / H, hh = bh - bb * H;
      for (int row0 = t * 128; row0 < min(N, t * 128 + 128); row0 += R::kRows) {  // stages without a row are left out
        if (!(ok = mbar_wait_warp(empty(s), ph ^ 1, w, kPSiteProducer))) break;
        const int rows = min(R::kRows, N - row0);
        if (lane == 0) {
          // a tiled copy delivers all rows of its box, zeros beyond the last one
          const uint32_t dense_bytes = rows * row_bytes, box_bytes = R::kRows * row_bytes;
          mbar_arrive_expect_tx(full(s), (so.n == d8 ? dense_bytes : box_bytes) + (sdo.n == d8 ? dense_bytes : box_bytes));
#pragma unroll
          for (int which = 0; which < 2; ++which) {
            const Strides& st = which ? sdo : so;
            const uint32_t dst = base + s * R::kStageBytes + which * R::kPartBytes;
            if (st.n == d8)
              bulk_load_1d(dst, (which ? dout : o) + bb * st.b + hh * st.h + static_cast<long long>(row0) * st.n,
                           dense_bytes, full(s));
            else
              tma_load_4d(dst, which ? &tdo : &to, 0, row0, HeadCoord{static_cast<int>(hh), static_cast<int>(bb)},
                          full(s));
          }
        }
        if (++s == R::kStages) s = 0, ph ^= 1;
      }
    }
    return;
  }

  // ---------------- consumer warps ----------------
  const int sub = threadIdx.x % kLanesPerRow;
  const int row_in_pass = threadIdx.x / kLanesPerRow;
  float lse_cur[kTilePasses], lse_nxt[kTilePasses];
  auto fetch_lse = [&](long long tile, float* dst) {
    const long long bh = tile / ntiles;
    const int t = static_cast<int>(tile - bh * ntiles);
#pragma unroll
    for (int i = 0; i < kTilePasses; ++i) {
      const int row = t * 128 + i * kRowsPerPass + row_in_pass;
      dst[i] = (sub == 0 && tile < tiles && row < N) ? ld_global(lse + bh * N + row) : INFINITY;
    }
  };
  fetch_lse(blockIdx.x, lse_cur);
  int it = 0, s = 0, ph = 0;
  long long prev_tile = -1;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
    fetch_lse(tile + gridDim.x, lse_nxt);
    const int t = static_cast<int>(tile % ntiles);
    const int tile_rows = min(128, N - t * 128);
    const int cb = it & 1;
    unsigned amax2 = 0;  // two running maxima of 15-bit magnitudes, one per 16-bit half
#pragma unroll
    for (int part = 0; part < R::kParts; ++part) {
      const int rows = tile_rows - part * R::kRows;  // of this stage, as far as it goes
      const bool staged = part == 0 || rows > 0;
      if (staged) {
        const bool ok = mbar_wait(full(s), ph, w, kPSiteConsumer);
        if (!consumers_all(ok, R::kConsumers)) return;
      }
      // the previous tile's results are complete in shared memory: one coalesced store
      if (part == 0 && prev_tile >= 0) {
        const int pb = (it - 1) & 1;
        rowstats[prev_tile * 256 + threadIdx.x] = stat[pb * 256 + threadIdx.x];
        if (threadIdx.x == 0) {
          unsigned m = wmax[pb * 8];
#pragma unroll
          for (int i = 1; i < 8; ++i) m = max(m, wmax[pb * 8 + i]);
          tile_amax[prev_tile] = m;
        }
      }
      const uint4* so_ = reinterpret_cast<const uint4*>(smem + s * R::kStageBytes);
      const uint4* sdo_ = reinterpret_cast<const uint4*>(smem + s * R::kStageBytes + R::kPartBytes);
      uint4 a[kPasses], b[kPasses];
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        const int r = i * kRowsPerPass + row_in_pass;
        if (r < rows && sub < d8) {
          a[i] = so_[r * d8 + sub];
          b[i] = sdo_[r * d8 + sub];
        } else {
          a[i] = make_uint4(0, 0, 0, 0);
          b[i] = make_uint4(0, 0, 0, 0);
        }
      }
      // Products and maxima first: the stage is given back once every piece has been used, not when
      // its load has been issued (an arrive can overtake a load that is still in flight).
      float dot[kPasses];
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        dot[i] = dot8<BF16>(a[i], b[i]);
        amax2 = __vmaxu2(amax2, b[i].x & 0x7fff7fffu);
        amax2 = __vmaxu2(amax2, b[i].y & 0x7fff7fffu);
        amax2 = __vmaxu2(amax2, b[i].z & 0x7fff7fffu);
        amax2 = __vmaxu2(amax2, b[i].w & 0x7fff7fffu);
        dot[i] += __shfl_xor_sync(0xffffffffu, dot[i], kLanesPerRow / 2);
      }
      __syncwarp();
      if (staged) {
        if (lane == 0) mbar_arrive(empty(s));
        if (++s == R::kStages) s = 0, ph ^= 1;
      }
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        float acc = dot[i];
#pragma unroll
        for (int off = kLanesPerRow / 4; off > 0; off >>= 1)
          acc += __shfl_xor_sync(0xffffffffu, acc, off);
        const int r = i * kRowsPerPass + row_in_pass;
        if (sub == 0) {
          const bool valid = r < rows;
          stat[cb * 256 + part * R::kRows + r] = valid ? -lse_cur[part * kPasses + i] * kLog2e : -INFINITY;
          stat[cb * 256 + 128 + part * R::kRows + r] = valid ? -acc : 0.f;
        }
      }
    }
    // largest magnitude of the tile: halves, warp, block (a NaN or inf pattern wins, which
    // head_dscale treats as "do not scale")
    unsigned m = max(amax2 & 0xffffu, amax2 >> 16);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) wmax[cb * 8 + warp] = m;
#pragma unroll
    for (int i = 0; i < kTilePasses; ++i) lse_cur[i] = lse_nxt[i];
    prev_tile = tile;
  }
  if (prev_tile >= 0) {
    named_bar_sync(1, R::kConsumers);
    const int pb = (it - 1) & 1;
    rowstats[prev_tile * 256 + threadIdx.x] = stat[pb * 256 + threadIdx.x];
    if (threadIdx.x == 0) {
      unsigned m = wmax[pb * 8];
#pragma unroll
      for (int i = 1; i < 8; ++i) m = max(m, wmax[pb * 8 + i]);
      tile_amax[prev_tile] = m;
    }
  }
}

// One thread converts 8 consecutive head-dim elements of one row.  Consecutive lanes take
// consecutive rows of the same 32-row group, so the fp32 reads are contiguous 512-byte runs
// (the layout the fused backward kernel accumulates into).
template <int D, bool BF16>
__global__ void __launch_bounds__(256)
    dq_convert_kernel(const float4* acc, uint4* __restrict__ dq, F32Out dq32, int N, int ntiles,
                      long long total, int d8, int H, Strides sdq) {
  grid_wait_previous();
  grid_allow_next();
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  // idx = ((tile_global * 4 + w) * (D/8) + k8) * 32 + lane
  const int lane = static_cast<int>(idx & 31);
  long long t = idx >> 5;
  const int k8 = static_cast<int>(t % (D / 8));
  t /= (D / 8);
  const int w = static_cast<int>(t & 3);
  const long long tile_global = t >> 2;
  const long long bh = tile_global / ntiles;
  const int tile = static_cast<int>(tile_global - bh * ntiles);
  const int row = tile * 128 + w * 32 + lane;
  if (row >= N || k8 >= d8) return;  // padding rows / padding columns of the accumulator
  const long long blk = (tile_global * 4 + w) * (D / 4);  // in units of [32 lanes][float4]
  const float4 x = ld_global(acc + (blk + 2 * k8) * 32 + lane);
  const float4 y = ld_global(acc + (blk + 2 * k8 + 1) * 32 + lane);
  const long long bb = bh / H, hh = bh - bb * H;
  if (dq32.p != nullptr) {
    const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    st_global_8(dq32.p + bb * dq32.st.b + hh * dq32.st.h + row * dq32.st.n + k8 * 8, v);
    return;
  }
  uint4 r;
  r.x = pack2<BF16>(x.x, x.y);
  r.y = pack2<BF16>(x.z, x.w);
  r.z = pack2<BF16>(y.x, y.y);
  r.w = pack2<BF16>(y.z, y.w);
  dq[bb * sdq.b + hh * sdq.h + row * sdq.n + k8] = r;  // strides in 16-byte units
}

// Element strides -> strides in 16-byte pieces (every stride is a multiple of 8 elements).
Strides in_vec8(const Strides& st) { return Strides{st.b / 8, st.h / 8, st.n / 8}; }

template <int D, bool BF16>
cudaError_t launch_pre_t(const AttnShape& s, const CUtensorMap& to, const CUtensorMap& tdo, const void* o,
                         const Strides& so, const void* dout, const Strides& sdo, const float* lse, float* rowstats, int* status,
                         int num_sms, cudaStream_t stream) {
  const int ntiles = (s.N + 127) / 128;
  const long long tiles = static_cast<long long>(s.B) * s.H * ntiles;
  unsigned* tile_amax = reinterpret_cast<unsigned*>(rowstats + tiles * 256);  // behind the last tile
  using R = PreRing<D>;
  auto* kernel = bwd_preprocess_ring_kernel<D, BF16>;
  const cudaError_t attr = cudaFuncSetAttribute(
      kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, R::kSmemBytes);
  if (attr != cudaSuccess) return attr;
  const unsigned grid = static_cast<unsigned>(tiles < num_sms ? tiles : num_sms);
  return launch_dependent(
      kernel, grid, R::kThreads, R::kSmemBytes, stream, to, tdo, static_cast<const uint4*>(o),
      static_cast<const uint4*>(dout), lse, rowstats, tile_amax,
      s.N, ntiles, tiles, s.Dg / 8, s.H, in_vec8(so), in_vec8(sdo), status);
}

template <int D, bool BF16>
cudaError_t launch_cvt_t(const AttnShape& s, const float* dq_accum, void* dq, const Strides& sdq,
                         const F32Out& dq32, cudaStream_t stream) {
  const int ntiles = (s.N + 127) / 128;
  const long long total = static_cast<long long>(s.B) * s.H * ntiles * 128 * (D / 8);
  const long long blocks = (total + 255) / 256;
  return launch_dependent(
      dq_convert_kernel<D, BF16>, static_cast<unsigned>(blocks), 256, 0, stream,
      reinterpret_cast<const float4*>(dq_accum), static_cast<uint4*>(dq), dq32, s.N, ntiles, total,
      s.Dg / 8, s.H, in_vec8(sdq));
}

}  // namespace

cudaError_t launch_bwd_preprocess(const AttnShape& s, const CUtensorMap& to, const CUtensorMap& tdo,
                                  const void* o, const Strides& so, const void* dout, const Strides& sdo, const float* lse,
                                  float* rowstats, int* status, int num_sms,
                                  cudaStream_t stream) {
#define FA2_CASE(DD)                                                                          \
  case DD:                                                                                    \
    return s.dtype                                                                            \
               ? launch_pre_t<DD, true>(s, to, tdo, o, so, dout, sdo, lse, rowstats, status, num_sms,  \
                                        stream)                                               \
               : launch_pre_t<DD, false>(s, to, tdo, o, so, dout, sdo, lse, rowstats, status, num_sms, \
                                         stream);
  switch (s.D) {
    FA2_CASE(32)
    FA2_CASE(64)
    FA2_CASE(128)
    FA2_CASE(256)
  }
#undef FA2_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_dq_convert(const AttnShape& s, const float* dq_accum, void* dq,
                              const Strides& sdq, const F32Out& dq32, cudaStream_t stream) {
#define FA2_CASE(DD)                                                        \
  case DD:                                                                  \
    return s.dtype ? launch_cvt_t<DD, true>(s, dq_accum, dq, sdq, dq32, stream)   \
                   : launch_cvt_t<DD, false>(s, dq_accum, dq, sdq, dq32, stream);
  switch (s.D) {
    FA2_CASE(32)
    FA2_CASE(64)
    FA2_CASE(128)
  }
#undef FA2_CASE
  return cudaErrorInvalidValue;
}

}  // namespace fa2
