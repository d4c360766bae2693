// One decoding step through a stack of transformer blocks: the host side of the whole stack in one call.
//
// A step of a small model is launch-bound: from Python a block took about 400 us of host time for 11 launches
// (24 blocks of width 1024: 9.1 ms per token against 1.7 ms of kernels).  Here a block is eight launches (norm, QKV,
// rotary + cache append, attention, output projection, norm, first MLP layer with its activation, second MLP layer)
// issued back to back from C++, each as a programmatic dependent of the one before, so launch latency and the first
// loads of the weights overlap the previous kernel's tail.  The first kernel of the stack is an ordinary launch:
// whatever wrote the weights or the cache before is complete, which is what lets the others read ahead.
#include "common.cuh"
#include <string.h>

namespace {

// z = norm(x0 (+ residual)), x_out = x0 + residual; one row per CTA, the row stays in registers (h <= 8192).
template <bool RMS>
__global__ void __launch_bounds__(256)
decode_norm_kernel(const __nv_bfloat16* x0, const __nv_bfloat16* residual, const __nv_bfloat16* __restrict__ gamma,
                   const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* z, __nv_bfloat16* x_out, int h, float eps) {
  constexpr int VPT = 4;
  __shared__ float red[2][8];
  mb::let_next_kernel_start();
  const size_t row = static_cast<size_t>(blockIdx.x) * h;
  const int nvec = h >> 3;
  mb::bf16x8 g[VPT], bt[VPT], xp[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + 256 * i;
    if (v < nvec) {
      g[i] = reinterpret_cast<const mb::bf16x8*>(gamma)[v];
      if (!RMS && beta) bt[i] = reinterpret_cast<const mb::bf16x8*>(beta)[v];
    }
  }
  mb::wait_for_previous_kernel();
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + 256 * i;
    if (v < nvec) {
      xp[i] = reinterpret_cast<const mb::bf16x8*>(x0 + row)[v];
      float x[8];
      mb::unpack8(xp[i], x);
      if (residual) {
        float r[8];
        mb::unpack8(reinterpret_cast<const mb::bf16x8*>(residual + row)[v], r);
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] += r[k];
        xp[i] = mb::pack8(x);
        mb::unpack8(xp[i], x);
      }
      reinterpret_cast<mb::bf16x8*>(x_out + row)[v] = xp[i];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        s += x[k];
        ss += x[k] * x[k];
      }
    }
  }
  s = mb::warp_sum(s);
  ss = mb::warp_sum(ss);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = s;
    red[1][w] = ss;
  }
  __syncthreads();
  s = ss = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s += red[0][j];
    ss += red[1][j];
  }
  const float mean = RMS ? 0.f : s / h;
  const float rstd = rsqrtf(fmaxf(ss / h - mean * mean, 0.f) + eps);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + 256 * i;
    if (v < nvec) {
      float x[8], gg[8], o[8], b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      mb::unpack8(xp[i], x);
      mb::unpack8(g[i], gg);
      if (!RMS && beta) mb::unpack8(bt[i], b);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = (x[k] - mean) * rstd * gg[k] + b[k];
      reinterpret_cast<mb::bf16x8*>(z + row)[v] = mb::pack8(o);
    }
  }
}

int launch_norm(const void* x0, const void* residual, const void* gamma, const void* beta, void* z, void* x_out,
                int rows, int h, float eps, int rms, int pdl, cudaStream_t stream) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(rows, 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  typedef const __nv_bfloat16* In;
  typedef __nv_bfloat16* Out;
  return cudaLaunchKernelEx(&cfg, rms ? decode_norm_kernel<true> : decode_norm_kernel<false>, static_cast<In>(x0),
                            static_cast<In>(residual), static_cast<In>(gamma), static_cast<In>(beta),
                            static_cast<Out>(z), static_cast<Out>(x_out), h, eps) == cudaSuccess
             ? 0
             : -4;
}

// Pointers of one block, in the order the caller fills them in; absent biases are null.
struct Block {
  const void *norm1_w, *norm1_b, *wqkv, *bqkv, *wo, *bo, *norm2_w, *norm2_b, *w1, *b1, *w2, *b2;
  void* cache;      // [>= batch][max_seq][2][hk][d]
};

}  // namespace

MB_API int mb_gemm_skinny_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                               int flags, const void* bias, const void* aux, float alpha, int always, int pdl,
                               cudaStream_t stream);
MB_API int mb_decode_attn(const void* q, const void* k, const void* v, void* o, int batch, int nh, int nh_kv, int d,
                          int len, long q_sb, long k_sb, long k_ss, long k_sh, long v_sb, long v_ss, long v_sh,
                          float scale, int pdl, cudaStream_t stream);
MB_API int mb_rope_append(void* qkv, void* cache, const float* cosv, const float* sinv, int batch, int seq, int hq,
                          int hk, int d, int rot, int off, long cache_sb, int pdl, cudaStream_t stream);

// Scratch that mb_decode_stack needs, in bf16 elements.
MB_API long mb_decode_stack_scratch(int batch, int h, int hq, int hk, int d, int f) {
  return static_cast<long>(batch) * (3L * h + (hq + 2L * hk) * d + static_cast<long>(hq) * d + f);
}

// hidden: [batch][h], the stack's input; residual may be null (the stream starts at the stack's input).  Writes the
// last block's MLP output to out_hidden and the residual stream in front of it to out_residual (their sum is what the
// next norm takes).  flags of the first MLP layer: 2 GELU, 128 SwiGLU.  off: position of the new token.  Every bf16
// pointer 16-byte aligned; h, f, hq * d, hk * d multiples of 8; h <= 8192, batch <= 128.  Returns the number of
// kernels launched, or a negative code.
MB_API int mb_decode_stack(const void* hidden, const void* residual, void* out_hidden, void* out_residual,
                           const void* blocks, int nblocks, void* scratch, int batch, int h, int hq, int hk, int d,
                           int f, int act_flags, int rms, float eps, const float* scale, const float* cosv,
                           const float* sinv, int rot, int off, long cache_sb, cudaStream_t stream) {
  if (batch <= 0 || batch > 128 || h % 8 || h > 8192 || f % 8 || nblocks <= 0) return -1;
  if ((act_flags & 128) && f % 64) return -1;
  const Block* bl = static_cast<const Block*>(blocks);
  __nv_bfloat16* z = static_cast<__nv_bfloat16*>(scratch);
  const long bh = static_cast<long>(batch) * h, qkv_cols = (hq + 2L * hk) * d;
  __nv_bfloat16* res_mid = z + bh;            // stream between attention and MLP
  __nv_bfloat16* branch = res_mid + bh;       // attention branch's output
  __nv_bfloat16* qkv = branch + bh;
  __nv_bfloat16* ctx = qkv + batch * qkv_cols;
  __nv_bfloat16* act = ctx + static_cast<long>(batch) * hq * d;
  const int ctx_cols = hq * d;
  int n = 0;
  const void* x = hidden;
  const void* res = residual;
#define MB_STEP(call)                       \
  do {                                      \
    const int rc_ = (call);                 \
    if (rc_ != 0) return rc_ < 0 ? rc_ : -9; \
    ++n;                                    \
  } while (0)
  for (int i = 0; i < nblocks; ++i) {
    const Block& b = bl[i];
    // the residual stream alternates between res_mid (behind norm1) and out_residual (behind norm2)
    MB_STEP(launch_norm(x, res, b.norm1_w, b.norm1_b, z, res_mid, batch, h, eps, rms, i > 0, stream));
    MB_STEP(mb_gemm_skinny_bf16(z, b.wqkv, qkv, batch, static_cast<int>(qkv_cols), h, h, h, static_cast<int>(qkv_cols),
                                b.bqkv ? 1 : 0, b.bqkv, nullptr, 1.f, 1, 1, stream));
    MB_STEP(mb_rope_append(qkv, b.cache, cosv, sinv, batch, 1, hq, hk, d, rot, off, cache_sb, 1, stream));
    const __nv_bfloat16* kc = static_cast<const __nv_bfloat16*>(b.cache);
    const __nv_bfloat16* vc = kc + static_cast<long>(hk) * d;
    MB_STEP(mb_decode_attn(qkv, kc, vc, ctx, batch, hq, hk, d, off + 1, qkv_cols, cache_sb, 2L * hk * d, d, cache_sb,
                           2L * hk * d, d, scale[i], 1, stream));
    MB_STEP(mb_gemm_skinny_bf16(ctx, b.wo, branch, batch, h, ctx_cols, ctx_cols, ctx_cols, h, b.bo ? 1 : 0, b.bo,
                                nullptr, 1.f, 1, 1, stream));
    MB_STEP(launch_norm(branch, res_mid, b.norm2_w, b.norm2_b, z, out_residual, batch, h, eps, rms, 1, stream));
    MB_STEP(mb_gemm_skinny_bf16(z, b.w1, act, batch, f, h, h, h, f, act_flags | (b.b1 ? 1 : 0), b.b1, nullptr, 1.f, 1, 1,
                                stream));
    MB_STEP(mb_gemm_skinny_bf16(act, b.w2, out_hidden, batch, h, f, f, f, h, b.b2 ? 1 : 0, b.b2, nullptr, 1.f, 1, 1,
                                stream));
    x = out_hidden;
    res = out_residual;
  }
#undef MB_STEP
  return n;
}
