// Device-side helpers shared by the data-plane kernels: system-scope
// flag load/store, bounded waits, 16-byte vector access, dtype conversion.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "eux_kernels.h"

namespace eux {

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint64_t ld_acquire_sys(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys(uint64_t* p, uint64_t v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Behind a __threadfence_system() of the same thread this publishes as a release store does. Every release store is a
// system-scope fence of its own, which waits for the store before it: a microsecond or more where that one goes to
// pinned host memory.
__device__ __forceinline__ void st_relaxed_sys(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_sys_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// What this thread has written or seen, other CTAs' work that it has counted included, before what it writes next, for this
// GPU and for everyone.
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void fence_sys() { asm volatile("fence.acq_rel.sys;" ::: "memory"); }
__device__ __forceinline__ void red_release_gpu_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Programmatic dependent launch, which takes the 2 to 2.5 us between the end of one kernel of a stream and the first load of
// the next away: what follows may be launched once every CTA has called this (a kernel that waits for another GPU or stream
// does not: what it lets in would hold SMs for as long). What is let in sits on the SMs until this kernel ends, where kernels
// of other streams find no room, so a CTA calls it when it has no more work to begin: the launch is through before the last
// tile is (called at the start, 8192^3 let a transfer of its stream hold up those of others for 0.7 ms, and calls in a loop
// were no faster: 128 x 8192 x 8192 bf16 30.2 and 30.3 us, 640 x 4096 x 1024 11.7 and 11.6) ...
__device__ __forceinline__ void allow_next_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// ... and a kernel launched so waits here until everything before it in the stream is complete and visible, before it touches
// memory. (Nothing to wait for in a plain launch.)
__device__ __forceinline__ void wait_for_launch_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The launch of a kernel that calls wait_for_launch_before.
template <typename... Args>
static inline int launch_early(void (*kernel)(Args...), int grid, int threads, size_t smem, cudaStream_t st, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid), cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, args...);
}

// The kernel's shared memory limit, raised before its first launch on a device to the most that any launch takes (threads
// that race do it twice). Set to each launch's own size, a smaller launch of another thread could lower it in between.
template <auto KERNEL>
static cudaError_t allow_smem(int dev, size_t most) {
  static std::atomic<bool> done[64];
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (done[dev].load(std::memory_order_acquire)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (e == cudaSuccess) done[dev].store(true, std::memory_order_release);
  return e;
}

// Spin until *flag >= value. Gives up after timeout_ns (0 = 2 s default) or
// 2^31 polls, whichever comes first; returns false on give-up.
__device__ __forceinline__ bool wait_flag_ge(const uint64_t* flag, uint64_t value, uint64_t timeout_ns) {
  if (ld_acquire_sys(flag) >= value) return true;
  const uint64_t limit = timeout_ns ? timeout_ns : 2000000000ull;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 0; it < 0x7fffffffu; ++it) {
    if (ld_acquire_sys(flag) >= value) return true;
    if ((it & 63u) == 63u) {
      if (globaltimer_ns() - t0 > limit) return false;
      __nanosleep(32);
    }
  }
  return false;
}
__device__ __forceinline__ bool wait_u32_ge_gpu(const uint32_t* flag, uint32_t value, uint64_t timeout_ns) {
  if (ld_acquire_gpu(flag) >= value) return true;
  const uint64_t limit = timeout_ns ? timeout_ns : 2000000000ull;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 0; it < 0x7fffffffu; ++it) {
    if (ld_acquire_gpu(flag) >= value) return true;
    if ((it & 63u) == 63u) {
      if (globaltimer_ns() - t0 > limit) return false;
      __nanosleep(32);
    }
  }
  return false;
}

__device__ __forceinline__ void set_status(uint32_t* status, uint32_t code, uint32_t where) {
  if (status) atomicCAS(status, 0u, code | (where << 8));
}

// 16-byte accesses that bypass L1 (data may have been written by another GPU).
__device__ __forceinline__ uint4 ld_cg_u4(const void* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ld_stream_u4(const void* p) {
  uint4 v;
  asm volatile("ld.global.cs.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void st_u4(void* p, uint4 v) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void st_stream_u4(void* p, uint4 v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

__host__ __device__ __forceinline__ int dtype_size(int dt) {
  switch (dt) {
    case EUX_DT_F32: return 4;
    case EUX_DT_F16: return 2;
    case EUX_DT_BF16: return 2;
    default: return 1;
  }
}

__device__ __forceinline__ float load_as_float(const void* base, uint64_t idx, int dt) {
  switch (dt) {
    case EUX_DT_F32: return reinterpret_cast<const float*>(base)[idx];
    case EUX_DT_F16: return __half2float(reinterpret_cast<const __half*>(base)[idx]);
    case EUX_DT_BF16: return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[idx]);
    case EUX_DT_F8E4M3: {
      __nv_fp8_e4m3 v;
      v.__x = reinterpret_cast<const uint8_t*>(base)[idx];
      return float(v);
    }
    default: return float(reinterpret_cast<const uint8_t*>(base)[idx]);
  }
}
__device__ __forceinline__ void store_from_float(void* base, uint64_t idx, int dt, float f) {
  switch (dt) {
    case EUX_DT_F32: reinterpret_cast<float*>(base)[idx] = f; break;
    case EUX_DT_F16: reinterpret_cast<__half*>(base)[idx] = __float2half_rn(f); break;
    case EUX_DT_BF16: reinterpret_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(f); break;
    case EUX_DT_F8E4M3: reinterpret_cast<uint8_t*>(base)[idx] = __nv_fp8_e4m3(f).__x; break;
    default: reinterpret_cast<uint8_t*>(base)[idx] = (uint8_t)f; break;
  }
}
__device__ __forceinline__ float apply_op(float x, int op, float arg) {
  return op == EUX_OP_ADD ? x + arg : (op == EUX_OP_MUL ? x * arg : x);
}

}  // namespace eux
