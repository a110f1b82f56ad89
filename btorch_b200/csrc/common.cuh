// Shared device/host helpers for the btorch_b200 kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <vector>

#include "../../include/btorch_b200.h"

// Set the thread-local error text and return `status` (defined in layout.cpp).
extern "C" int bt_set_error(int status, const char* fmt, ...);

#define BT_CHECK_ARG(cond, ...)                                  \
  do {                                                           \
    if (!(cond)) return bt_set_error(BT_ERR_INVALID, __VA_ARGS__); \
  } while (0)

// Report a failed launch (configuration errors surface here, asynchronous
// faults surface at the caller's next synchronisation).
#define BT_CHECK_LAUNCH(what)                                              \
  do {                                                                     \
    cudaError_t err_ = cudaGetLastError();                                 \
    if (err_ != cudaSuccess)                                               \
      return bt_set_error(BT_ERR_CUDA, "%s: %s", what, cudaGetErrorString(err_)); \
  } while (0)

namespace bt {

constexpr int kWarp = 32;
constexpr uint32_t kIdMask = (1u << BT_BIN_SHIFT) - 1u;

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Single-rounding IEEE fp32 operations.  The intrinsics are never fused into
// FMA by the compiler, so the device evaluates exactly the rounding sequence of
// the reference's eager CPU operators (one rounding per torch op).
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }

__device__ __forceinline__ float ld(const bt_param& p, int64_t i) { return __ldg(p.ptr + i * p.stride); }

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

// L2 eviction-priority hints (PTX createpolicy + .L2::cache_hint, sm_80+).
// Data read once per step (edge lists, the step's input current) is loaded
// evict-first so that it does not push the small, reused accumulators out of
// L2; reductions into those accumulators are issued evict-last.
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_evict_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_evict_normal() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// Loads that bring the whole 128-byte line into L2: what follows is read soon.
__device__ __forceinline__ uint2 ld_nc_u2_line(const void* ptr, uint64_t pol) {
  uint2 v;
  asm("ld.global.nc.L2::cache_hint.L2::128B.v2.u32 {%0, %1}, [%2], %3;" : "=r"(v.x), "=r"(v.y) : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ uint4 ld_nc_u4_line(const void* ptr, uint64_t pol) {
  uint4 v;
  asm("ld.global.nc.L2::cache_hint.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ int32_t ld_nc_s32_line(const int32_t* ptr) {
  int32_t v;
  asm("ld.global.nc.L2::128B.s32 %0, [%1];" : "=r"(v) : "l"(ptr));
  return v;
}
// Read-only (non-coherent) loads with an L2 policy; not volatile, so the
// compiler may batch them ahead of their uses.
__device__ __forceinline__ uint4 ld_nc_u4(const void* ptr, uint64_t pol) {
  uint4 v;
  asm("ld.global.nc.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ uint2 ld_nc_u2(const void* ptr, uint64_t pol) {
  uint2 v;
  asm("ld.global.nc.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;" : "=r"(v.x), "=r"(v.y) : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ uint32_t ld_nc_u32(const void* ptr, uint64_t pol) {
  uint32_t v;
  asm("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_nc_f32(const float* ptr, uint64_t pol) {
  float v;
  asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(ptr), "l"(pol));
  return v;
}
// Coherent fp32 load / store with an L2 policy.
__device__ __forceinline__ float ld_f32(const float* ptr, uint64_t pol) {
  float v;
  asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ void st_f32(float* ptr, float v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(ptr), "f"(v), "l"(pol) : "memory");
}
// 16-byte loads / stores of four consecutive floats with an L2 policy.
__device__ __forceinline__ float4 ld_nc_f4(const float* ptr, uint64_t pol) {
  float4 v;
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ float4 ld_f4(const float* ptr, uint64_t pol) {
  float4 v;
  asm volatile("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ void st_f4(float* ptr, float4 v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(ptr), "f"(v.x), "f"(v.y),
               "f"(v.z), "f"(v.w), "l"(pol)
               : "memory");
}
// fp32 reduction (no return value) with an L2 policy.
__device__ __forceinline__ void red_add_f32(float* ptr, float v, uint64_t pol) {
  // no "memory" clobber: nothing in the issuing kernel reads the target, so
  // independent loads may be scheduled across the reduction
  asm volatile("red.global.add.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(ptr), "f"(v), "l"(pol));
}

// SMs of the current device.
inline int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
    (void)cudaGetLastError();
    return 148;
  }
  return sms;
}

// Launch set-ups already checked (kernel, device, dynamic shared memory,
// blocks): the attribute calls and occupancy queries of a persistent launch
// run once per set-up, not on every call -- they cost the host far more
// than a short launch takes on the device.
struct LaunchSetup {
  const void* kern;
  int dev;
  size_t smem;
  int blocks;
};
inline std::mutex& launch_setup_mutex() {
  static std::mutex m;
  return m;
}
inline std::vector<LaunchSetup>& launch_setups() {
  static std::vector<LaunchSetup> v;
  return v;
}
inline bool launch_setup_known(const void* kern, int dev, size_t smem, int blocks) {
  std::lock_guard<std::mutex> g(launch_setup_mutex());
  for (const LaunchSetup& e : launch_setups())
    if (e.kern == kern && e.dev == dev && e.smem == smem && e.blocks == blocks) return true;
  return false;
}
// The dynamic shared memory to allow a kernel: at least `smem` and never less
// than a set-up already checked on this device asked for (the attribute is
// the kernel's, shared by all its set-ups).
inline size_t launch_smem_allow(const void* kern, int dev, size_t smem) {
  std::lock_guard<std::mutex> g(launch_setup_mutex());
  for (const LaunchSetup& e : launch_setups())
    if (e.kern == kern && e.dev == dev && e.smem > smem) smem = e.smem;
  return smem;
}
inline void launch_setup_add(const void* kern, int dev, size_t smem, int blocks) {
  std::lock_guard<std::mutex> g(launch_setup_mutex());
  launch_setups().push_back(LaunchSetup{kern, dev, smem, blocks});
}

// Programmatic dependent launch of the step kernels: a launch may be scheduled
// as soon as every block of the one before it has started (step_begin signals
// it), so its launch latency and the set-up of its blocks overlap the other's
// tail; step_begin then waits for that grid to complete and its writes to be
// visible before any global access.
// A block may thus be resident while the launch before its own, and even the
// one before that, still writes.  So:
//  - the first launch of a chain is an ordinary one (first): all that was
//    written before the chain is complete when any of its blocks starts, and
//    may be read through the read-only path and ahead of the wait;
//  - what a launch of the chain writes (state, spike sets and lists, transposed
//    operands, packed weights) is read by the later ones through plain pointers:
//    no __restrict__, __ldg, __ldcg or ld.global.nc, whose loads need data that
//    does not change while the kernel is resident and are not ordered after
//    the wait.
__device__ __forceinline__ void step_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The wait alone: the next launch starts when this one's blocks have left.  The
// neuron step of the scatter takes it: with delivery blocks resident beside it, steps in
// which half of the neurons fire were slower (4000 neurons, 40 samples, 5 bins, 256
// steps: 38.0 ms with the early start, 32.3 without, 33.7 before there was any;
// 65536 neurons, 40 samples: 92.7, 85.5, 85.9), quiet ones as fast within 2 %.
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_step(bool first, void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = first ? 0 : 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace bt
