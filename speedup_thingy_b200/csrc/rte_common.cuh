// Shared device/host helpers for the rte_b200 kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "rte_b200.h"

#define RTE_CHECK_ARG(cond) \
  do {                      \
    if (!(cond)) return RTE_ERR_BAD_ARG; \
  } while (0)

#define RTE_LAUNCH_CHECK()                                   \
  do {                                                       \
    cudaError_t e__ = cudaPeekAtLastError();                 \
    if (e__ != cudaSuccess) return RTE_ERR_LAUNCH;           \
  } while (0)

// Device status codes written to the caller's status word.
enum : int {
  RTE_DEV_WAIT_TIMEOUT_PRODUCER = 101,
  RTE_DEV_WAIT_TIMEOUT_MMA = 102,
  RTE_DEV_WAIT_TIMEOUT_EPILOGUE = 103,
  RTE_DEV_WAIT_TIMEOUT_PEER = 104,
  RTE_DEV_INDEX_OUT_OF_RANGE = 201,
  RTE_DEV_CAPACITY_OVERFLOW = 202
};

namespace rte {

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline long long ceil_div64(long long a, long long b) { return (a + b - 1) / b; }

// Programmatic dependent launch: a kernel launched with the attribute may start while the kernel before it in the stream
// still runs.  grid_dependency_wait returns once that kernel has completed and its writes are visible (at once without the
// attribute); nothing the kernel before may touch is read or written ahead of it.  grid_dependents_launch lets the next
// such kernel begin its own set-up.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void after_previous_grid() { grid_dependency_wait(); grid_dependents_launch(); }

// Launches a kernel that begins with after_previous_grid() so that its start overlaps the end of the kernel before it.
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);      // (an error stays pending for RTE_LAUNCH_CHECK)
}

// Where a call of rte_router_aux_bwd_data(dh0 = NULL) leaves the parts of d pooled in its scratch, and their add into every
// token's gradient (router.cu).
inline const float* router_dpooled(const float* scratch, int B, int hid, int R, int K) {
  return scratch + (((size_t)RTE_ROUTER_MAX_R + (size_t)B * (2 * hid + R + K) + 3) & ~(size_t)3);
}
int add_router_dpooled(float* dh0, const float* dpooled, int B, int S, int d, cudaStream_t st);

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum; `red` is shared scratch of >= 32 floats.  All threads get the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? red[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

__device__ __forceinline__ float silu_f(float g) { return g / (1.f + __expf(-g)); }
__device__ __forceinline__ float sigmoid_f(float g) { return 1.f / (1.f + __expf(-g)); }

// SiLU and sigmoid of the fused epilogues of large products: 1 / (1 + 2^(-g log2 e)) with the approximate ex2 and rcp of the PTX ISA, four
// instructions and no slow path for huge denominators (a correctly rounded divide's stalls the whole epilogue warp; __expf with
// __fdividef, which give the same for all 2^32 arguments, take 80.0 us instead of 76 for 16384 x 512 -> 2048).  Relative error up to
// (4 + 2 |g|) 2^-24 for g > -64, most of it the exponential's (all arguments compared with 64 bits; with a correctly rounded
// quotient (3.5 + 2 |g|) 2^-24); 0 below -87.3, where the denominator passes 2^126.  What they go into is rounded to bf16.
__device__ __forceinline__ float fast_sigmoid(float g) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  return r;
}
__device__ __forceinline__ float fast_silu(float g) { return g * fast_sigmoid(g); }

// The bits of sigmoid_f and silu_f without the branches of their divide: an approximate reciprocal, then a step with fused multiply-adds
// that corrects the quotient by its remainder (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990).  A quarter of the denominator keeps the approximation out of the range that it flushes; maximum and minimum
// take the place of infinity * 0.  Compared with sigmoid_f for all 2^32 arguments; silu_of_bf16 with silu_f for all bf16 ones
// (of the others, two of 2^32 differ in the last bit).
__device__ __forceinline__ float quarter_rcp(float y) {          // about 1 / y
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(0.25f * y));
  return 0.25f * r;
}
__device__ __forceinline__ float sigmoid_rn(float g) {
  const float y = 1.f + __expf(-g), r = quarter_rcp(y);
  return __fmaf_rn(fmaxf(__fmaf_rn(-y, r, 1.f), -1.f), r, r);
}
__device__ __forceinline__ float silu_of_bf16(float g) {
  const float y = 1.f + __expf(-g), r = quarter_rcp(y), q = g * r;
  return __fmaf_rn(-fminf(__fmaf_rn(y, q, -g), 3.40282347e38f), r, q);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
__device__ __forceinline__ float bf16_to_f(const __nv_bfloat16* p) { return __bfloat162float(*p); }

}  // namespace rte
