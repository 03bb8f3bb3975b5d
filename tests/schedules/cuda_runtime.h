// Host stand-in for the CUDA headers the kernels include, and for the helpers of ptx.cuh: the barrier
// operations go to the scheduler in main.cpp, everything that only moves data does nothing.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __grid_constant__
#define __restrict__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)
#define asm
#define volatile(...)  // `asm volatile(...)` vanishes; `volatile int*` stays

struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct uint4 { unsigned x, y, z, w; };
struct dim3 {
  unsigned x, y, z;
  dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {}
};
inline float2 make_float2(float x, float y) { return {x, y}; }
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return {x, y, z, w}; }
struct alignas(64) CUtensorMap { char bytes[128]; };
using cudaStream_t = void*;
enum cudaError_t { cudaSuccess, cudaErrorInvalidValue };
enum { cudaLaunchAttributeProgrammaticStreamSerialization, cudaFuncAttributeMaxDynamicSharedMemorySize };
struct cudaLaunchAttribute {
  int id;
  struct { int programmaticStreamSerializationAllowed; } val;
};
struct cudaLaunchConfig_t {
  dim3 gridDim, blockDim;
  size_t dynamicSmemBytes;
  cudaStream_t stream;
  cudaLaunchAttribute* attrs;
  int numAttrs;
};
template <typename F>
cudaError_t cudaFuncSetAttribute(F*, int, int) { return cudaSuccess; }

// One lane (lane 0) stands for each warp.
extern dim3 threadIdx, blockIdx, gridDim;
extern uint8_t* sim_smem;
void sim_arrive(uint32_t bar);
void sim_arrive_later(uint32_t bar);      // a copy's bytes arrive at some later time
void sim_arrive_after_mma(uint32_t bar);  // behind everything in the in-order tensor pipe
void sim_init(uint32_t bar, uint32_t count);
bool sim_wait(uint32_t bar, uint32_t parity, int site, volatile int* abort_flag, bool vote);  // false: given up
void __syncthreads();
void sim_wait_previous();
void sim_access();  // of global memory: not before the kernel has waited for its predecessor
void sim_stored(int row);  // of an output
void sim_run(unsigned warps, void (*body)(void*), void* arg);

template <typename... Params, typename... Args>
cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* cfg, void (*kernel)(Params...), Args&&... args) {
  auto body = [&] { kernel(args...); };
  gridDim = cfg->gridDim;
  for (unsigned b = 0; b < cfg->gridDim.x; ++b) {
    blockIdx = dim3(b, 0, 0);
    sim_run(cfg->blockDim.x / 32, [](void* p) { (*static_cast<decltype(body)*>(p))(); }, &body);
  }
  return cudaSuccess;
}

inline void __syncwarp() {}
bool sim_meet(bool x);  // false, too, when a lane may have left with false
inline bool __all_sync(unsigned, bool x) { return sim_meet(x); }
inline bool __any_sync(unsigned, bool x) { return x; }
inline unsigned __reduce_max_sync(unsigned, unsigned x) { return x; }
template <typename T> T atomicAdd(T* p, T v) { T old = *p; *p += v; return old; }
template <typename T> T atomicExch(T* p, T v) { T old = *p; *p = v; return old; }
template <typename T> T atomicCAS(T* p, T cmp, T v) { T old = *p; if (old == cmp) *p = v; return old; }
inline float __uint_as_float(unsigned x) { float f; memcpy(&f, &x, 4); return f; }
inline unsigned __float_as_uint(float f) { unsigned x; memcpy(&x, &f, 4); return x; }
inline float2 __ffma2_rn(float2, float2, float2) { return {0, 0}; }
inline float2 __fadd2_rn(float2, float2) { return {0, 0}; }
inline float2 __fmul2_rn(float2, float2) { return {0, 0}; }
using std::max;
using std::min;
inline unsigned max(int a, unsigned b) { return std::max<unsigned>(a, b); }

namespace fa2 {
struct HeadCoord { int h, b; };
struct WaitCtx {
  volatile int* abort_flag;
  int* status;
};
constexpr uint32_t kSwizzle128B = 2, kSwizzle64B = 4;
template <bool BF16> constexpr bool kInterBF16 = BF16;
constexpr uint32_t make_idesc_ab(int, int, bool, bool, bool, bool) { return 0; }
constexpr uint32_t make_idesc(int, int, bool, bool, bool) { return 0; }
inline uint32_t smem_u32(const void* p) { return uint32_t(static_cast<const uint8_t*>(p) - sim_smem); }
inline uint32_t elect_one() { return 1; }
inline void mbar_init(uint32_t bar, uint32_t count) { sim_init(bar, count); }
inline void mbar_arrive(uint32_t bar) { sim_arrive(bar); }
inline void mbar_arrive_expect_tx(uint32_t bar, uint32_t) { sim_access(), sim_arrive_later(bar); }
inline void mma_commit(uint32_t bar) { sim_arrive_after_mma(bar); }
inline bool mbar_wait(uint32_t bar, uint32_t parity, const WaitCtx& w, int site) { return sim_wait(bar, parity, site, w.abort_flag, false); }
inline bool mbar_wait_warp(uint32_t bar, uint32_t parity, const WaitCtx& w, int site) { return sim_wait(bar, parity, site, w.abort_flag, true); }
template <typename T> T ld_global(const T* p) { return sim_access(), *p; }
inline void tmem_ld_x32(uint32_t, uint32_t* r) { memset(r, 0, 128); }
inline void tmem_ld_x16(uint32_t, uint32_t* r) { memset(r, 0, 64); }
template <bool BF16> uint32_t pack2(float, float) { return 0; }
inline float2 ex2_poly2(float2 x) { return x; }
inline float ex2(float) { return 0; }
inline float lg2(float) { return 0; }
inline float max3(float, float, float) { return 0; }
#define FA2_NOTHING(name) template <typename... A> void name(A&&...) {}
FA2_NOTHING(fence_mbar_init) FA2_NOTHING(fence_proxy_async_smem) FA2_NOTHING(tma_load_4d) FA2_NOTHING(bulk_load_1d)
FA2_NOTHING(tma_store_commit) FA2_NOTHING(tma_store_wait_all) FA2_NOTHING(tma_store_wait_read)
FA2_NOTHING(prefetch_tensormap) FA2_NOTHING(tmem_alloc) FA2_NOTHING(tmem_relinquish) FA2_NOTHING(tmem_dealloc)
FA2_NOTHING(tc_fence_before) FA2_NOTHING(tc_fence_after) FA2_NOTHING(tmem_wait_ld) FA2_NOTHING(tmem_wait_st)
FA2_NOTHING(tmem_st_x32) FA2_NOTHING(tmem_st_x16) FA2_NOTHING(mma_ss) FA2_NOTHING(mma_ts) FA2_NOTHING(st_global_8)
FA2_NOTHING(grid_allow_next)
inline void tma_store_4d(const CUtensorMap*, int, int row, HeadCoord, uint32_t) { sim_stored(row); }
inline void grid_wait_previous() { sim_wait_previous(); }
template <int N> void reg_inc() {}
template <int N> void reg_dec() {}
}  // namespace fa2
