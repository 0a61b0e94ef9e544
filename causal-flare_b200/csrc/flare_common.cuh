// Shared device/host helpers for the FLARE B200 kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/flare_b200.h"

namespace flare {

constexpr float kNegInf = -INFINITY;

// ---------------------------------------------------------------------------------------------
// host-side error plumbing
// ---------------------------------------------------------------------------------------------
void set_cuda_error(cudaError_t e, const char* where);

#define FLARE_CUDA_CHECK(expr)                         \
  do {                                                 \
    cudaError_t _e = (expr);                           \
    if (_e != cudaSuccess) {                           \
      ::flare::set_cuda_error(_e, #expr);              \
      return FLARE_ERR_CUDA;                           \
    }                                                  \
  } while (0)

int sm_count();

// Per-kernel timing for callers that ask for a profile (the reference's profile=True returns one entry per kernel
// launch, causal_flare/autoregressive/training.py:4-50).  While switched on (flare_profile_enable) every launch site
// brackets its kernel with a pair of CUDA events on the launch stream; flare_profile_entry reads them back.
struct LaunchTimer {
  LaunchTimer(const char* name, cudaStream_t stream);
  ~LaunchTimer();
  int slot;
  cudaStream_t stream;
};

// Programmatic dependent launch: the kernels of a call follow one another on the stream, most of them for a few
// microseconds or (the standby kernels) for no time at all.  Every kernel launched here waits (pdl_wait) until the kernels
// before it have completed and their writes are visible before it touches anything, so nothing is read or written earlier
// than in a plain launch; only the launch latencies overlap.  The short kernels let the next kernel of the stream be set up
// as soon as they start (pdl_begin), the tensor-core backward when a CTA has fetched its last tile, the tensor-core forward
// and the walk that stands by behind it when they end (no trigger).  CTAs of the next kernel that wait on the GPU slow the
// forward down (B=8 N=8192 H=16 M=128 D=64: 188.7 us triggered at the start, 185.2 us at its last tile, 183.5 us at its end),
// and a forward whose CTAs are placed while the walk of the call before still drains runs slower from its first chunk to its
// last (causal B=2 N=65536 H=32 M=256 D=128 back to back: 2192 us with a trigger in the walk, 2066 us without).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_trigger();
  pdl_wait();
}
// What a kernel reads may have been written by the kernel before it, which can still be running when this one starts.  So no
// load goes through the read-only path (which assumes memory that nobody writes while the kernel runs, and whose loads the
// compiler may move over the wait): no __restrict__ inputs, no read-only intrinsics; and the streaming loads below are pinned
// behind the wait like it.
__device__ __forceinline__ float4 load_streaming(const float4* p) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 load_streaming(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

constexpr int kMaxDynamicSmem = 227 * 1024;  // what a block may have beyond the system's own kilobyte

// Allows a kernel (one without static shared memory) all the dynamic shared memory there is.  Always the same limit, whatever
// the launch at hand needs: a kernel's limit is shared by all host threads, and one that lowered it for its own launch would
// fail another's.  Asked for on every launch: the limit belongs to the context, which the host may have torn down and rebuilt
// since the last call.
template <typename Kern>
inline cudaError_t allow_smem(Kern kern) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
}

// While one lives, the forwards that this thread plans take no more workspace for segment states than fits `bytes` (for
// callers that cannot supply what flare_forward_workspace_bytes asks for).
struct ScratchLimit {
  explicit ScratchLimit(size_t bytes);
  ~ScratchLimit();
  ScratchLimit(const ScratchLimit&) = delete;
  size_t before;
};

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

inline int dtype_size(int dtype) { return dtype == FLARE_F32 ? 4 : 2; }

// ---------------------------------------------------------------------------------------------
// runtime-typed element access (dtype is uniform per launch, so these branches never diverge)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float bf16_bits_to_float(uint32_t bits16) { return __uint_as_float(bits16 << 16); }

// Load 8 consecutive elements starting at element index `off` (off % 8 == 0, base 16-byte aligned).
__device__ __forceinline__ void load8(const void* base, int dtype, int64_t off, float (&out)[8]) {
  if (dtype == FLARE_F32) {
    const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + off);
    float4 a = *p, b = *(p + 1);
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
    out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
  } else {
    const uint4 r = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + off);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
    if (dtype == FLARE_BF16) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        out[2 * i] = bf16_bits_to_float(w[i] & 0xffffu);
        out[2 * i + 1] = bf16_bits_to_float(w[i] >> 16);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __half2 h = *reinterpret_cast<const __half2*>(&w[i]);
        const float2 f = __half22float2(h);
        out[2 * i] = f.x;
        out[2 * i + 1] = f.y;
      }
    }
  }
}

__device__ __forceinline__ float load1(const void* base, int dtype, int64_t off) {
  if (dtype == FLARE_F32) return reinterpret_cast<const float*>(base)[off];
  if (dtype == FLARE_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[off]);
  return __half2float(reinterpret_cast<const __half*>(base)[off]);
}

__device__ __forceinline__ void store1(void* base, int dtype, int64_t off, float x) {
  if (dtype == FLARE_F32) reinterpret_cast<float*>(base)[off] = x;
  else if (dtype == FLARE_BF16) reinterpret_cast<__nv_bfloat16*>(base)[off] = __float2bfloat16_rn(x);
  else reinterpret_cast<__half*>(base)[off] = __float2half_rn(x);
}

// Store 4 consecutive elements (off % 4 == 0, base 16-byte aligned).
__device__ __forceinline__ void store4(void* base, int dtype, int64_t off, float a, float b, float c, float d) {
  if (dtype == FLARE_F32) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + off) = make_float4(a, b, c, d);
  } else if (dtype == FLARE_BF16) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    uint2 r;
    r.x = *reinterpret_cast<uint32_t*>(&lo);
    r.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + off) = r;
  } else {
    __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
    uint2 r;
    r.x = *reinterpret_cast<uint32_t*>(&lo);
    r.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + off) = r;
  }
}

// ---------------------------------------------------------------------------------------------
// score transforms
// ---------------------------------------------------------------------------------------------
// sigma(x) = (1+x)^p for x >= 0, (1-x)^-p for x < 0.
__device__ __forceinline__ float stablemax_sigma(float x, float p) {
  const float base = 1.0f + fabsf(x);
  float r;
  if (p == 1.0f) r = base;
  else if (p == 2.0f) r = base * base;
  else if (p == 3.0f) r = base * base * base;
  else if (p == 4.0f) { const float b2 = base * base; r = b2 * b2; }
  else r = exp2f(p * log2f(base));
  return x >= 0.0f ? r : 1.0f / r;
}

// sigma'(x) / sigma(x) = p / (1 + |x|) on both branches.
__device__ __forceinline__ float stablemax_slope_ratio(float x, float p) { return p / (1.0f + fabsf(x)); }

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace flare
