// Shared device helpers for the sm_100a kernel library.
//
// Everything in this library is exported with C linkage and takes raw device
// pointers plus a cudaStream_t, so the Python side binds it with ctypes and no
// framework headers are needed at build time.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#define MB_API extern "C" __attribute__((visibility("default")))

// Status words written by kernels whose waits can give up.  The host reads the
// word after the launch; a non-zero value means the kernel returned early.
enum MbStatus : int {
  MB_OK = 0,
  MB_ERR_TIMEOUT_FULL = 1,     // consumer gave up waiting for a TMA stage
  MB_ERR_TIMEOUT_EMPTY = 2,    // producer gave up waiting for a free stage
  MB_ERR_TIMEOUT_TMEM = 3,     // epilogue / MMA gave up waiting for an accumulator
  MB_ERR_TIMEOUT_PEER = 4,     // a flag written by another rank never arrived
  MB_ERR_BAD_ARG = 5,
};

namespace mb {

constexpr int kWarp = 32;

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

// Block-wide reductions through shared memory; `red` needs 32 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = (lane < nw) ? red[lane] : 0.f;
  r = warp_sum(r);
  return r;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = (lane < nw) ? red[lane] : -INFINITY;
  r = warp_max(r);
  return r;
}

// Programmatic dependent launch: a kernel launched with the attribute may start once every CTA of the kernel before
// it has called let_next_kernel_start (or left), and sees that kernel's results after wait_for_previous_kernel.
// Both do nothing in an ordinary launch.  Data of the kernel before must not be read through const __restrict__
// pointers: the compiler may move such loads in front of the wait.
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void let_next_kernel_start() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// 16-byte vector of 8 bf16 values.
struct __align__(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ bf16x8 pack8(const float* f) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

// Two fp32 values in one 64-bit register: sm_100 issues one instruction for both (element 0 in the low half).
typedef uint64_t f32x2;
__device__ __forceinline__ f32x2 pack_f32x2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul_f32x2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add_f32x2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// bf16 pair -> fp32 pair (a bf16 is the upper half of an fp32)
__device__ __forceinline__ f32x2 bf16x2_to_f32x2(uint32_t p) {
  return pack_f32x2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}

// tanh on the special-function unit (max abs error ~5e-4, far below bf16 resolution).
__device__ __forceinline__ float fast_tanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * x * (1.f + k1 * x * x);
  return 0.5f * x * (1.f + fast_tanh(u));
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * x * (1.f + k1 * x * x);
  float t = fast_tanh(u);
  float du = k0 * (1.f + 3.f * k1 * x * x);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }

}  // namespace mb
