// Mixed-precision Adam / AdamW on a flat shard: fp32 master weights and moments,
// bf16 (or fp32) gradient in, bf16 model weights out, all in one pass.
//
// One launch does what the reference spreads over three: the grad cast to fp32
// (mist/re_swap_manager/optimizer.py:514-518), apex multi_tensor_adam with
// inv_scale (mist/optimizers/fused_adam.py:583-690) and the master -> model
// cast-copy (mist/re_swap_manager/optimizer.py:571-599).
#include "common.cuh"

namespace {

struct AdamArgs {
  float lr, beta1, beta2, eps, weight_decay;
  float bias_c1, bias_c2;  // 1 - beta^t
  float inv_scale;         // gradients are multiplied by this first (loss scale, 1/dp, ...)
  int adamw;               // 1: decoupled weight decay, 0: L2 added to the gradient
};

// Eight fp32 values, every byte touched once and by one pass only: 32-byte accesses (whole sectors) that leave L1 alone
// where the array allows it, two of 16 bytes otherwise.
template <bool WIDE>
__device__ __forceinline__ void load8(const float* src, float* f) {
  if (WIDE) {
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
                 : "l"(src));
  } else {
    const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
}
template <bool WIDE>
__device__ __forceinline__ void load8(const __nv_bfloat16* src, float* f) {
  mb::unpack8(*reinterpret_cast<const mb::bf16x8*>(src), f);
}
template <bool WIDE>
__device__ __forceinline__ void store8(float* dst, const float* f) {
  if (WIDE) {
    asm volatile("st.global.L1::no_allocate.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(dst), "f"(f[0]),
                 "f"(f[1]), "f"(f[2]), "f"(f[3]), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7])
                 : "memory");
  } else {
    reinterpret_cast<float4*>(dst)[0] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4*>(dst)[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

__device__ __forceinline__ void adam_update(float& p, float& m, float& v, float g,
                                            const AdamArgs& a) {
  g *= a.inv_scale;
  if (!a.adamw) g += a.weight_decay * p;
  m = a.beta1 * m + (1.f - a.beta1) * g;
  v = a.beta2 * v + (1.f - a.beta2) * g * g;
  float mh = m / a.bias_c1;
  float vh = v / a.bias_c2;
  float upd = mh / (sqrtf(vh) + a.eps);
  if (a.adamw) upd += a.weight_decay * p;
  p -= a.lr * upd;
}

// Bound by memory: 28 bytes an element.  One vector of eight per thread and no loop, so that the loads of a CTA that
// starts overlap the stores of those that end: 80 M elements 361 -> 329 us (6.2 -> 6.8 TB/s; before: a grid of 16 CTAs
// per SM that looped, 16-byte accesses).
template <typename GradT, bool WIDE>
__global__ void __launch_bounds__(256)
adam_kernel(float* __restrict__ master, float* __restrict__ exp_avg, float* __restrict__ exp_avg_sq,
            const GradT* __restrict__ grad, __nv_bfloat16* __restrict__ model, size_t n,
            AdamArgs a) {
  const size_t nvec = n >> 3;
  const size_t i = blockIdx.x * static_cast<size_t>(256) + threadIdx.x;
  if (i < nvec) {
    float g[8], p[8], m[8], v[8];
    load8<WIDE>(grad + 8 * i, g);
    load8<WIDE>(master + 8 * i, p);
    load8<WIDE>(exp_avg + 8 * i, m);
    load8<WIDE>(exp_avg_sq + 8 * i, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) adam_update(p[k], m[k], v[k], g[k], a);
    store8<WIDE>(master + 8 * i, p);
    store8<WIDE>(exp_avg + 8 * i, m);
    store8<WIDE>(exp_avg_sq + 8 * i, v);
    if (model) reinterpret_cast<mb::bf16x8*>(model)[i] = mb::pack8(p);
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 7)) {
    size_t j = (nvec << 3) + threadIdx.x;
    float p = master[j], m = exp_avg[j], v = exp_avg_sq[j];
    adam_update(p, m, v, static_cast<float>(grad[j]), a);
    master[j] = p;
    exp_avg[j] = m;
    exp_avg_sq[j] = v;
    if (model) model[j] = __float2bfloat16(p);
  }
}

}  // namespace

// All arrays hold `n` elements and must be 16-byte aligned (32 for the wide accesses).  `model` may be null.
MB_API int mb_adam_step(float* master, float* exp_avg, float* exp_avg_sq, const void* grad,
                        int grad_is_fp32, void* model, size_t n, float lr, float beta1, float beta2,
                        float eps, float weight_decay, int step, float inv_scale, int adamw,
                        cudaStream_t stream) {
  if (!n) return 0;
  AdamArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.weight_decay = weight_decay;
  a.bias_c1 = 1.f - powf(beta1, static_cast<float>(step));
  a.bias_c2 = 1.f - powf(beta2, static_cast<float>(step));
  a.inv_scale = inv_scale;
  a.adamw = adamw;
  const size_t nvec = (n + 7) / 8;
  const size_t blocks = (nvec + 255) / 256;
  if (blocks > 0x7fffffff) return -1;
  const uintptr_t all = reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(exp_avg) |
                        reinterpret_cast<uintptr_t>(exp_avg_sq) | (grad_is_fp32 ? reinterpret_cast<uintptr_t>(grad) : 0);
  const bool wide = (all & 31) == 0;
#define MB_ADAM(T_, W_)                                                                                      \
  adam_kernel<T_, W_><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(                                    \
      master, exp_avg, exp_avg_sq, reinterpret_cast<const T_*>(grad), reinterpret_cast<__nv_bfloat16*>(model), n, a)
  if (grad_is_fp32) { if (wide) MB_ADAM(float, true); else MB_ADAM(float, false); }
  else { if (wide) MB_ADAM(__nv_bfloat16, true); else MB_ADAM(__nv_bfloat16, false); }
#undef MB_ADAM
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
