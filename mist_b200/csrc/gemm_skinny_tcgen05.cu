// bf16 linear layer for a handful of tokens (decoding, short prompts):
//
//   y[M, N] = epi(x[M, K] W[N, K]^T),  M <= 128        epi: + bias, GELU, + residual, or SwiGLU over [gate | up]
//
// Bound: reading W once from HBM.  The ordinary GEMM tiles put the tokens on the 128-row side of the MMA and give a
// CTA 128 columns of W, so a 4096 x 4096 layer ran on 32 CTAs of 148 (39 us for 33.6 MB, 0.9 TB/s).  Here
//   * W is the 128-row operand and the tokens are the 16 .. 128 columns, so no MMA row is padding;
//   * the CTAs of a cluster (up to eight) share the K range of a tile and sum their fp32 partial tiles through
//     distributed shared memory in rank order: enough CTAs for any N, one launch, no workspace, the same bits on
//     every run;
//   * four stages keep W streaming: 18 - 24 KB each and two or three CTAs per SM up to 64 tokens (150 - 220 KB in
//     flight), 32 KB each and one CTA per SM (128 KB) above;
//   * W does not depend on the kernel before: launched as a programmatic dependent (`pdl`), the CTAs start to load W
//     while that kernel drains and wait for it only before they read x.  The caller may ask for that only where no
//     kernel still running can write W.
// Warps: 0 TMA, 1 MMA, 2 - 5 read the accumulator; all six finish the outputs.
//
// Reference counterpart: the cuBLAS calls of csrc/fused_dense_lib/fused_dense_cuda.cu:19-92 at small batch.
#include "sm100_pair.cuh"
#include <string.h>
#include <type_traits>

using namespace sm100;

namespace {

constexpr int BR = 128;       // rows of W per CTA (64 gate + 64 up rows in the SwiGLU form)
constexpr int BK = 64;
constexpr int kThreads = 192;
constexpr int kStages = 4;
constexpr int kMaxSplit = 8;

enum EpiFlags : int { EPI_BIAS = 1, EPI_GELU = 2, EPI_RESIDUAL = 64, EPI_SWIGLU = 128 };

struct SkinnyParams {
  int M, N, K;               // N: output columns
  __nv_bfloat16* C;
  int ldc;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* aux;  // residual, [M][N] with row stride ldc
  int flags;
  float alpha;
  int* status;
};

template <int NT>
struct SkinnyLayout {
  static constexpr int kW = BR * BK * 2;
  static constexpr int kX = NT * BK * 2;
  static constexpr int kStage = kW + kX;
  static constexpr int kPartStride = BR + 4;                      // floats per token of the partial tile
  static constexpr int kPart = NT * kPartStride * 4;              // over the stages, once they have been read
  static constexpr int kRing = kStages * kStage;
  static constexpr int kBarOffset = kRing > kPart ? kRing : kPart;
  static constexpr int kTotal = kBarOffset + (2 * kStages + 1) * 8 + 16;
};

__device__ __forceinline__ void report(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}
// (volatile keeps the load behind the cluster barrier; without a memory clobber several can be in flight)
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}

template <int NT>
__global__ void __launch_bounds__(kThreads)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x,
                   const SkinnyParams p) {
  using L = SkinnyLayout<NT>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* done_bar = empty_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = gridDim.x, rank = blockIdx.x;
  const bool swiglu = (p.flags & EPI_SWIGLU) != 0;
  const int width = swiglu ? BR / 2 : BR;            // output columns of this tile
  const int n0 = blockIdx.y * width;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = static_cast<int>(static_cast<long>(num_kb) * rank / split);
  const int kb1 = static_cast<int>(static_cast<long>(num_kb) * (rank + 1) / split);
  constexpr int kTmemCols = NT < 32 ? 32 : NT;

  mb::let_next_kernel_start();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    prefetch_tmap(&tma_w);
    prefetch_tmap(&tma_x);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      uint32_t armed[kStages];
      for (int s = 0; s < kStages; ++s) armed[s] = 0;
      const int row_a = n0, row_b = swiglu ? p.N + n0 : n0 + BR / 2;
      auto load_w = [&](int i) {
        const int s = i % kStages;
        uint8_t* sw = smem + s * L::kStage;
        mbar_expect_tx(&full_bar[s], L::kStage);
        armed[s]++;
        tma_load_2d(sw, &tma_w, &full_bar[s], (kb0 + i) * BK, row_a);
        tma_load_2d(sw + L::kW / 2, &tma_w, &full_bar[s], (kb0 + i) * BK, row_b);
      };
      auto load_x = [&](int i) {
        const int s = i % kStages;
        tma_load_2d(smem + s * L::kStage + L::kW, &tma_x, &full_bar[s], (kb0 + i) * BK, 0);
      };
      const int n = kb1 - kb0, head = n < kStages ? n : kStages;
      for (int i = 0; i < head; ++i) load_w(i);
      mb::wait_for_previous_kernel();
      for (int i = 0; i < head; ++i) load_x(i);
      for (int i = head; i < n; ++i) {
        if (!mbar_wait(&empty_bar[i % kStages], ((i / kStages) - 1) & 1)) {
          report(p.status, MB_ERR_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        load_w(i);
        load_x(i);
      }
      if (!ok) {      // gave up: let the copies already in flight land before the CTA exits
        for (int s = 0; s < kStages; ++s)
          if (armed[s]) mbar_wait(&full_bar[s], (armed[s] - 1) & 1, 50);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(BR, NT, 0, 0);
    bool ok = true;
    for (int i = 0; i < kb1 - kb0; ++i) {
      const int s = i % kStages;
      if (!mbar_wait(&full_bar[s], (i / kStages) & 1)) {
        report(p.status, MB_ERR_TIMEOUT_FULL);
        ok = false;
        break;
      }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t sw = smem_u32(smem + s * L::kStage), sx = sw + L::kW;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          mma_f16_ss(tmem_base, make_smem_desc_sw128(sw + k * 32, 16, 1024), make_smem_desc_sw128(sx + k * 32, 16, 1024),
                     idesc, (i | k) != 0 ? 1u : 0u);
        mma_commit(&empty_bar[s]);
      }
      __syncwarp();
    }
    if (ok && elect_one()) mma_commit(done_bar);
    __syncwarp();
  } else {
    const int q = warp & 3, r = q * 32 + lane;       // accumulator lane = row of W
    float* part = reinterpret_cast<float*>(smem);
    if (mbar_wait(done_bar, 0)) {                    // every MMA has read its stage: the ring is free
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < NT / 16; ++c) {
        uint32_t a[16];
        tmem_ld16(tmem_base + c * 16 + (static_cast<uint32_t>(q * 32) << 16), a);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) part[(c * 16 + i) * L::kPartStride + r] = __uint_as_float(a[i]);
      }
    } else {
      report(p.status, MB_ERR_TIMEOUT_TMEM);
    }
  }
  mb::wait_for_previous_kernel();       // this thread may read the residual and overwrite C below
  tc_fence_before();
  __syncthreads();
  if (split > 1) cluster_sync_all();

  // Four neighbouring columns per thread, the same ones for all of its tokens; the CTAs of the cluster take the tokens in
  // turn.
  // The loads of two tokens (and of all parts) are issued before the first sum: with one pair of columns at a time a
  // tile of 128 tokens spent 12 us here, 280 ns an output.
  const int quads = width / 4;                             // 32, or 16 for SwiGLU: both divide the threads
  const int c = (threadIdx.x % quads) * 4, n = n0 + c;
  const int live = min(4, p.N - n);                        // columns that exist; may be negative
  const int m_step = split * (kThreads / quads);
  if (live > 0) {
    float bias[4] = {0.f, 0.f, 0.f, 0.f}, bias_up[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.flags & EPI_BIAS) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < live) {
          bias[i] = __bfloat162float(p.bias[n + i]);
          if (swiglu) bias_up[i] = __bfloat162float(p.bias[p.N + n + i]);
        }
      }
    }
    const bool wide = live == 4 && (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & 7) == 0;
    const float* part = reinterpret_cast<const float*>(smem) + c;
    const uint32_t part_u = smem_u32(part);
    constexpr int U = 2;
    for (int m0 = rank + split * (threadIdx.x / quads); m0 < p.M; m0 += U * m_step) {
      float v[U][4], up[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int m = m0 + u * m_step;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (m >= p.M) {
        } else if (split == 1) {
          const float* at = part + m * L::kPartStride;
          a = *reinterpret_cast<const float4*>(at);
          if (swiglu) b = *reinterpret_cast<const float4*>(at + BR / 2);
        } else {
          const uint32_t off = part_u + static_cast<uint32_t>(m * L::kPartStride) * 4;
          float4 x[kMaxSplit], y[kMaxSplit];
#pragma unroll
          for (int r = 0; r < kMaxSplit; ++r) {
            x[r] = y[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < split) {
              const uint32_t at = map_to_cta(off, r);
              x[r] = ld_cluster4(at);
              if (swiglu) y[r] = ld_cluster4(at + (BR / 2) * 4);
            }
          }
#pragma unroll
          for (int r = 0; r < kMaxSplit; ++r) {
            a.x += x[r].x; a.y += x[r].y; a.z += x[r].z; a.w += x[r].w;
            b.x += y[r].x; b.y += y[r].y; b.z += y[r].z; b.w += y[r].w;
          }
        }
        v[u][0] = a.x; v[u][1] = a.y; v[u][2] = a.z; v[u][3] = a.w;
        up[u][0] = b.x; up[u][1] = b.y; up[u][2] = b.z; up[u][3] = b.w;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int m = m0 + u * m_step;
        if (m >= p.M) break;
        const long o = static_cast<long>(m) * p.ldc + n;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float x = v[u][i] * p.alpha;
          if (p.flags & EPI_BIAS) x += bias[i];
          if (p.flags & EPI_GELU) x = mb::gelu_tanh(x);
          if (swiglu) {
            float y = up[u][i] * p.alpha;
            if (p.flags & EPI_BIAS) y += bias_up[i];
            x = mb::silu(x) * y;
          }
          if ((p.flags & EPI_RESIDUAL) && i < live) x += __bfloat162float(p.aux[o + i]);
          v[u][i] = x;
        }
        if (wide) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(v[u][0], v[u][1]), hi = __floats2bfloat162_rn(v[u][2], v[u][3]);
          uint2 w;
          w.x = *reinterpret_cast<const uint32_t*>(&lo);
          w.y = *reinterpret_cast<const uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(p.C + o) = w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i < live) p.C[o + i] = __float2bfloat16(v[u][i]);
        }
      }
    }
  }
  if (split > 1) cluster_sync_all();      // nobody leaves while its partial tile is being read
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}
bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {BK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return encode_with_context([&] {
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}

template <int NT>
void skinny_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int tiles, int split, cudaStream_t stream) {
  memset(cfg, 0, sizeof(*cfg));
  cfg->gridDim = dim3(split, tiles, 1);
  cfg->blockDim = dim3(kThreads, 1, 1);
  cfg->dynamicSmemBytes = SkinnyLayout<NT>::kTotal + 1024;
  cfg->stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
}
template <int NT>
bool configure() {
  static const bool ok = cudaFuncSetAttribute(gemm_skinny_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              SkinnyLayout<NT>::kTotal + 1024) == cudaSuccess;
  return ok;
}
// SMs that clusters of a size can occupy together, one CTA on each (cudaOccupancyMaxActiveClusters on a B200: the CTAs of
// a cluster share a GPC).  A constant, so that sums are cut the same way on every GPU.
constexpr int kClusterSms[kMaxSplit + 1] = {0, 148, 148, 135, 132, 130, 132, 105, 120};

// CTAs that share a tile's K range: as many as leave each at least two K blocks and the whole grid resident
// (three CTAs per SM with 16 columns, one with 128, whose stages are larger): a second wave costs more than shorter sums
// give.  7680 x 2560 at 32 tokens (60 tiles): 4 CTAs a tile 11.7 us, 8 CTAs 19.4; 12288 x 4096 (96 tiles, at most 90
// clusters of three): 2 CTAs a tile 22.4 us, 3 CTAs 29.0; 22016 x 4096 at one token (172 tiles): 2 CTAs a tile 31.2 us,
// one 33.8.  Against at least four K blocks each, in a chain of launches of 1 - 128 tokens: 1024 x 1024 5.0 -> 4.6 us at one
// token and 8.4 -> 7.2 at 128, 512 x 512 4.6 -> 4.1 and 9.9 -> 7.8; the worst of 128 sizes 3072 x 1024 at 64 tokens, 7.1 -> 7.3.
// Sums of fewer than eight K blocks stay whole: 128 x 256 took 3.3 us in one part, 4.1 in two.
template <int NT>
int choose_split(int tiles, int num_kb) {
  constexpr int per_sm = NT == 16 ? 3 : NT <= 64 ? 2 : 1;
  if (num_kb < 8) return 1;
  int split = num_kb / 2 < kMaxSplit ? num_kb / 2 : kMaxSplit;
  while (split > 1 && kClusterSms[split] / split * per_sm < tiles) --split;
  return split < 1 ? 1 : split;
}

// Whether this kernel beats the tiled ones, which put the tokens on the 128-row side of the product; both sides measured
// for N from 64 to 50304 and K from 64 to 50304.  Up to 32 tokens it does at every size (0.14 - 0.96 of their time).
// Above, its epilogue needs enough K blocks to hide behind: at 64 tokens 512 x 512 took 7.5 us in two parts against 6.7 and
// 50304 x 1024 28.9 against 28.1, but 1024 x 1024 7.0 against 8.9.  Above 64 its stages leave one CTA per SM, and it has
// to split K to win: 128 tokens, 4096 x 4096 16 us against 24, but 12288 x 4096 31 against 26.
bool pays(int M, int num_kb, int split) {
  return M <= 32 || (split > 1 && num_kb >= 16) || (M <= 64 && num_kb >= 32);
}

template <int NT>
int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int tiles, int split, int pdl,
                  cudaStream_t stream) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  skinny_config<NT>(&cfg, attr, tiles, split, stream);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<NT>, tw, tx, p) == cudaSuccess ? 0 : -4;
}

}  // namespace

MB_API int* mb_status_device_ptr();

// C[M, N] = epi(alpha * A[M, K] B[N, K]^T) for M <= 128, bf16 in and out.  flags: bias, GELU, residual (aux, row
// stride ldc), or 128: SwiGLU, where B holds 2 N rows [gate | up] (and the bias 2 N values).  A and B 16-byte
// aligned, lda and ldb multiples of 8.  Returns 1 without launching when the arguments need another kernel or, unless
// `always`, when another one is faster.
MB_API int mb_gemm_skinny_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                               int flags, const void* bias, const void* aux, float alpha, int always, int pdl,
                               cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda & 7) || (ldb & 7) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15))
    return -1;
  if (M > 128 || (flags & ~(EPI_BIAS | EPI_GELU | EPI_RESIDUAL | EPI_SWIGLU)) || (reinterpret_cast<uintptr_t>(C) & 3))
    return 1;
  const bool swiglu = (flags & EPI_SWIGLU) != 0;
  if ((swiglu && (flags & EPI_GELU)) || ((flags & EPI_RESIDUAL) && !aux)) return 1;
  if (swiglu && N % (BR / 2)) return 1;      // a tile would mix gate rows with up rows
  const int width = swiglu ? BR / 2 : BR;
  const int tiles = (N + width - 1) / width;
  if (tiles > 65535) return 1;
  const int num_kb = (K + BK - 1) / BK;
  SkinnyParams p;
  p.M = M; p.N = N; p.K = K;
  p.C = reinterpret_cast<__nv_bfloat16*>(C);
  p.ldc = ldc;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.aux = reinterpret_cast<const __nv_bfloat16*>(aux);
  p.flags = flags;
  p.alpha = alpha;
  p.status = mb_status_device_ptr();
  auto run = [&](auto nt) -> int {
    constexpr int NT = decltype(nt)::value;
    if (!configure<NT>()) return -3;
    const int split = choose_split<NT>(tiles, num_kb);
    if (!always && !pays(M, num_kb, split)) return 1;
    CUtensorMap tw, tx;
    if (!make_map(&tw, B, static_cast<uint64_t>(N) * (swiglu ? 2 : 1), K, ldb, BR / 2)) return -2;
    if (!make_map(&tx, A, M, K, lda, NT)) return -2;
    return launch_skinny<NT>(tw, tx, p, tiles, split, pdl, stream);
  };
  if (M <= 16) return run(std::integral_constant<int, 16>());
  if (M <= 32) return run(std::integral_constant<int, 32>());
  if (M <= 64) return run(std::integral_constant<int, 64>());
  return run(std::integral_constant<int, 128>());
}
