// common.cuh -- shared helpers of the sm_100a GROG library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/pygrog_b200.h"

namespace pgb {

// ---- error reporting ------------------------------------------------------
void set_error(const char* fmt, ...);
void clear_error();

#define PGB_REQUIRE(cond, code, ...) \
  do {                               \
    if (!(cond)) {                   \
      ::pgb::set_error(__VA_ARGS__); \
      return (code);                 \
    }                                \
  } while (0)

// Launch check: returns PGB_ERR_CUDA from the enclosing function on failure.
#define PGB_LAUNCH_CHECK(name)                                                \
  do {                                                                        \
    cudaError_t e_ = cudaGetLastError();                                      \
    if (e_ != cudaSuccess) {                                                  \
      ::pgb::set_error("%s: launch failed: %s", name, cudaGetErrorString(e_)); \
      return PGB_ERR_CUDA;                                                    \
    }                                                                         \
  } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

constexpr int kNumSMs = 148;  // B200

// Number of the calling thread's current driver context, never given twice in a
// process (0: none yet, or the driver does not tell).
inline unsigned long long context_id() {
  using CtxGetId = int (*)(void*, unsigned long long*);
  static const CtxGetId get = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<CtxGetId>(fn);
    cudaGetLastError();
    return static_cast<CtxGetId>(nullptr);
  }();
  unsigned long long id = 0;
  return get != nullptr && get(nullptr, &id) == 0 ? id : 0;
}

// Lets kernel K take `bytes` of dynamic shared memory.  The call costs the host
// about a microsecond of a launch's five, so it is left out while the context is
// the one that K was last allowed it in (the limit belongs to a context: another
// device's, another one of this device, the one after cudaDeviceReset).
template <auto K>
inline void allow_smem(int bytes) {
  static std::atomic<unsigned long long> allowed{0};
  const unsigned long long ctx = context_id();
  if (ctx != 0 && allowed.load(std::memory_order_relaxed) == ctx) return;
  if (cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
    allowed.store(ctx, std::memory_order_relaxed);
}

// Launch that need not wait for the stream's previous kernel to be flushed
// before its blocks are placed (programmatic stream serialization): it hides
// part of the launch latency of short kernels in a row.  Such a kernel calls
// grid_wait() before its first access to global memory, which returns when the
// previous kernel is complete and its writes are visible.  The kernels do not
// trigger the next one early: its waiting blocks take their room (20 CG
// iterations at 128^2 / 30 at 320^2, us: 451 / 2173 plain, 433 / 2201 with an
// early trigger, 431 / 2167 without).
template <class... P, class... A>
inline cudaError_t launch_chained(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... a) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(a)...);
}
__device__ __forceinline__ void grid_wait() {
#ifdef __CUDA_ARCH__
  cudaGridDependencySynchronize();
#endif
}

inline int grid_for(int64_t n, int block, int64_t max_blocks = 148 * 32) {
  int64_t g = (n + block - 1) / block;
  if (g < 1) g = 1;
  if (g > max_blocks) g = max_blocks;
  return static_cast<int>(g);
}

// ---- complex arithmetic on float2 / double2 -------------------------------
template <typename R>
struct cplx;
template <>
struct cplx<float> {
  using T = float2;
};
template <>
struct cplx<double> {
  using T = double2;
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// acc += a * b
__device__ __forceinline__ void cfma(float2& acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.x = fmaf(-a.y, b.y, acc.x);
  acc.y = fmaf(a.x, b.y, acc.y);
  acc.y = fmaf(a.y, b.x, acc.y);
}
__device__ __forceinline__ void cfma(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}
// acc += conj(a) * b
__device__ __forceinline__ void cfma_conj(float2& acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.x = fmaf(a.y, b.y, acc.x);
  acc.y = fmaf(a.x, b.y, acc.y);
  acc.y = fmaf(-a.y, b.x, acc.y);
}
__device__ __forceinline__ void cfma_conj(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
}
template <typename V>
__device__ __forceinline__ V czero();
template <>
__device__ __forceinline__ float2 czero<float2>() {
  return make_float2(0.f, 0.f);
}
template <>
__device__ __forceinline__ double2 czero<double2>() {
  return make_double2(0.0, 0.0);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

__device__ __forceinline__ void catomic_add(float2* p, float2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}
__device__ __forceinline__ void catomic_add(double2* p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

// Warp-aggregated complex atomic add: lanes holding the same key are summed
// in registers first, then one lane per distinct key issues the atomic.
// Keys must be valid (>= 0) for all lanes in `active`.
template <typename V>
__device__ __forceinline__ void warp_aggregated_add(V* base, int64_t key, V val,
                                                    unsigned active) {
  unsigned peers = __match_any_sync(active, (unsigned long long)key);
  int leader = __ffs(peers) - 1;
  unsigned m = peers;
  V acc = czero<V>();
  while (m) {
    int src = __ffs(m) - 1;
    m &= m - 1;
    V v;
    v.x = __shfl_sync(peers, val.x, src);
    v.y = __shfl_sync(peers, val.y, src);
    acc = cadd(acc, v);
  }
  if ((int)(threadIdx.x & 31) == leader) catomic_add(base + key, acc);
}

__device__ __forceinline__ void warp_aggregated_add_real(float* base, int64_t key, float val,
                                                         unsigned active) {
  unsigned peers = __match_any_sync(active, (unsigned long long)key);
  int leader = __ffs(peers) - 1;
  unsigned m = peers;
  float acc = 0.f;
  while (m) {
    int src = __ffs(m) - 1;
    m &= m - 1;
    acc += __shfl_sync(peers, val, src);
  }
  if ((int)(threadIdx.x & 31) == leader) atomicAdd(base + key, acc);
}
__device__ __forceinline__ void warp_aggregated_add_real(double* base, int64_t key, double val,
                                                         unsigned active) {
  unsigned peers = __match_any_sync(active, (unsigned long long)key);
  int leader = __ffs(peers) - 1;
  unsigned m = peers;
  double acc = 0.0;
  while (m) {
    int src = __ffs(m) - 1;
    m &= m - 1;
    acc += __shfl_sync(peers, val, src);
  }
  if ((int)(threadIdx.x & 31) == leader) atomicAdd(base + key, acc);
}

}  // namespace pgb
