// Attention of one new query per sequence against a key/value cache (autoregressive decoding), and the step in
// front of it: rotary embedding of the new tokens' q and k with the append of k and v to the cache.
//
//   o[b, h, :] = softmax(scale * q[b, h, :] . K[b, 0:len, kv(h), :]) V[b, 0:len, kv(h), :]
//
// Bound: reading the cache once; there is no tensor-core work in a 1 x len product.  One CTA per (head, sequence)
// reached 0.17 TB/s on one sequence of 2048 positions (32 CTAs, one position in flight per warp: 193 us) and
// 1.6 TB/s on 32 sequences of 1000 (32 heads of 80; 201 us); this kernel takes 9.7 us and 57 us (5.7 TB/s), the other
// remains for short sequences (see short_is_faster).  Here
//   * a cluster of up to eight CTAs shares the positions of one (head, sequence) and merges its partial
//     (max, sum, output) triples through distributed shared memory: enough CTAs for one sequence, one launch,
//     no workspace;
//   * every warp streams its own positions through a ring of shared-memory stages with 16-byte asynchronous copies
//     (16 positions of head size 64, 8 of 80 - 128, 4 of 256 per stage, K and V; no barrier between warps): all 32
//     lanes copy whatever the head size, and two to three stages per warp are in flight while one is used.  Loads
//     into registers instead kept 41 KB per SM in flight and read 32 x 1000 positions at 2.4 TB/s;
//   * a position takes only the d / 8 lanes that hold a part of it, so a warp scores 32 / lanes positions at a
//     time.  With the copies in flight the kernel is bound by issue slots: 138 instructions per step of a plain
//     version took 115 us for 32 x 1000 positions of 32 x 80 (57 % of the slots).  So the four scores of a lane are
//     summed over the lanes together (each round halves what a lane still holds; a lane ends up with one score, one
//     maximum and one exponential per stage, and the four probabilities are handed out by shuffles), products run on
//     packed fp32 pairs, and the piece addresses advance by a constant;
//   * two CTAs fit an SM at every head size: what is merged lies over the ring, and a short chunk takes only the stages
//     that it fills.  With arrays of their own, and four stages at head size 64, one CTA fitted: 32 x 1000 positions of
//     32 heads of 128 on 8 took 119 us, now 32; 16 x 130 positions of 32 heads of 64 58 us, now 8.7;
//   * query heads that share a key/value head (grouped-query attention) go through one CTA in groups of up to
//     four, so the cache is read once per group of four instead of once per query head.
//
// Reference counterpart: csrc/ft_attention (FasterTransformer masked_multihead_attention,
// decoder_masked_multihead_attention_template.hpp:865; binding ft_attention.cpp:226), used by
// the inference path of mist/modules/mha.py:531-575.
#include "sm100_pair.cuh"
#include <limits.h>
#include <string.h>

#define BF(p) reinterpret_cast<const __nv_bfloat16*>(p)
#define BFM(p) reinterpret_cast<__nv_bfloat16*>(p)
#define LAUNCH_OK() (cudaGetLastError() == cudaSuccess ? 0 : -4)

namespace {

constexpr int kWarps = 8;
constexpr int kMaxD = 256;
constexpr int kUnroll = 4;         // steps of 32 / LPP positions per stage
constexpr int kMaxSplit = 8;      // largest portable cluster

__device__ __forceinline__ float ld_cluster(const float* p, uint32_t rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n"
               : "=f"(v)
               : "r"(sm100::map_to_cta(sm100::smem_u32(p), rank))
               : "memory");
  return v;
}

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}

// Maxima, sums and weighted values of the warps (s_) and of the CTA (c_).
template <int LPP, int G>
struct MergeArrays {
  float s_acc[kWarps][G][LPP * 8], c_acc[G][LPP * 8];
  float s_m[kWarps][G], s_l[kWarps][G], c_m[G], c_l[G];
};

// LPP lanes hold one position (a power of two >= d / 8), G query heads share the CTA.
template <int LPP, int G, int STAGES>
__global__ void __launch_bounds__(kWarps * 32, 2)
decode_attn_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, __nv_bfloat16* o, int nh,
                   int group, int d, int len, int chunk, int stages, long q_sb, long k_sb, long k_ss, long k_sh,
                   long v_sb, long v_ss, long v_sh, float scale_log2) {
  constexpr int PPW = 32 / LPP;
  constexpr int NP = PPW * kUnroll;         // positions per stage of a warp
  extern __shared__ __align__(16) uint8_t ring[];
  // what is merged lies over the ring, once every warp has read its positions
  using Merge = MergeArrays<LPP, G>;
  Merge& sm = *reinterpret_cast<Merge*>(ring);

  const int split = blockIdx.x, nsplit = gridDim.x;
  const int h0 = blockIdx.y * G, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPP;               // which of the warp's positions
  const int e0 = (lane % LPP) * 8;
  const bool live = e0 < d;                 // d is a multiple of 8, so a lane is all in or all out
  const int hk = h0 / group;

  const __nv_bfloat16* kb = k + b * k_sb + hk * k_sh;
  const __nv_bfloat16* vb = v + b * v_sb + hk * v_sh;

  // m: the same in all lanes of a position group; l: the lane's own probabilities only; acc: eight channels, in pairs
  float m[G], l[G];
  mb::f32x2 acc[G][4];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[g][i] = 0;
  }
  const int j0 = split * chunk, j1 = min(len, j0 + chunk);
  const int vph = d >> 3;                                     // 16-byte pieces of one head
  const int stage_elems = 2 * NP * d;                         // K rows, then V rows
  // [warp][stage]: a chunk that takes fewer than STAGES stages has only those, and never reaches a later one
  const __nv_bfloat16* wring = reinterpret_cast<const __nv_bfloat16*>(ring) + warp * stages * stage_elems;
  const uint32_t wring_u = sm100::smem_u32(wring);
  const int first = j0 + warp * NP;
  // the pieces this lane copies: NP * vph of K and as many of V, at most four of each per lane
  const __nv_bfloat16 *kp[4], *vp[4];
  int piece_row[4];
  uint32_t piece_at[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = lane + 32 * i, row = t / vph, col = (t - row * vph) * 8;
    piece_row[i] = row < NP ? first + row : INT_MAX;      // position of the piece; no position: past every end
    piece_at[i] = static_cast<uint32_t>(t) * 16;
    kp[i] = kb + static_cast<long>(first + row) * k_ss + col;
    vp[i] = vb + static_cast<long>(first + row) * v_ss + col;
  }
  const long k_step = static_cast<long>(kWarps * NP) * k_ss, v_step = static_cast<long>(kWarps * NP) * v_ss;
  uint32_t fetch_at = wring_u;
  int fetch_base = first, fetch_slot = 0;
  // copies the next stage; pieces past the end are filled with zeros and not read
  auto fetch = [&]() {
    if (fetch_base < j1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (static_cast<int>(piece_at[i]) < NP * d * 2) {
          const bool real = piece_row[i] < j1;
          copy16(fetch_at + piece_at[i], real ? kp[i] : kb, real);
          copy16(fetch_at + piece_at[i] + NP * d * 2, real ? vp[i] : vb, real);
          kp[i] += k_step;
          vp[i] += v_step;
          piece_row[i] += kWarps * NP;
        }
      }
    }
    fetch_base += kWarps * NP;
    fetch_at += stage_elems * 2;
    if (++fetch_slot == STAGES) {
      fetch_slot = 0;
      fetch_at = wring_u;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // As a dependent launch: the cache rows before the newest position were complete before the kernel in front of
  // this one started, so a CTA without that position begins to stream while that kernel drains.
  mb::let_next_kernel_start();
  if (j1 >= len) mb::wait_for_previous_kernel();
  const int steps = first < j1 ? (j1 - first + kWarps * NP - 1) / (kWarps * NP) : 0;
#pragma unroll
  for (int it = 0; it < STAGES - 1; ++it) fetch();
  mb::wait_for_previous_kernel();
  mb::f32x2 qf[G][4];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (live) raw = *reinterpret_cast<const uint4*>(q + b * q_sb + static_cast<long>(h0 + g) * d + e0);
    qf[g][0] = mb::bf16x2_to_f32x2(raw.x);
    qf[g][1] = mb::bf16x2_to_f32x2(raw.y);
    qf[g][2] = mb::bf16x2_to_f32x2(raw.z);
    qf[g][3] = mb::bf16x2_to_f32x2(raw.w);
  }
  // after the two exchange rounds of a score reduction a lane holds the score of step `mine`
  constexpr int O1 = LPP / 2, O2 = LPP / 4;
  const bool up1 = (lane & O1) != 0, up2 = (lane & O2) != 0;
  const int mine = (up1 ? 2 : 0) + (up2 ? 1 : 0);
  const int lane0 = lane & ~(O1 | O2);
  for (int it = 0; it < steps; ++it) {
    const int base = first + it * kWarps * NP;
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncwarp();                  // every lane's pieces of stage `it` are there, and everyone is done with it - 1
    fetch();
    const __nv_bfloat16* sk = wring + (it % STAGES) * stage_elems + sub * d + e0;
    const __nv_bfloat16* sv = sk + NP * d;
    float dot[G][kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      uint4 raw = make_uint4(0, 0, 0, 0);
      if (live) raw = *reinterpret_cast<const uint4*>(sk + u * PPW * d);
      const mb::f32x2 k0 = mb::bf16x2_to_f32x2(raw.x), k1 = mb::bf16x2_to_f32x2(raw.y),
                      k2 = mb::bf16x2_to_f32x2(raw.z), k3 = mb::bf16x2_to_f32x2(raw.w);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        mb::f32x2 s = mb::mul_f32x2(qf[g][0], k0);
        s = mb::fma_f32x2(qf[g][1], k1, s);
        s = mb::fma_f32x2(qf[g][2], k2, s);
        s = mb::fma_f32x2(qf[g][3], k3, s);
        const float2 t = mb::unpack_f32x2(s);
        dot[g][u] = t.x + t.y;
      }
    }
    const bool seen = base + mine * PPW + sub < j1;
    float prob[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float r0 = __shfl_xor_sync(0xffffffffu, up1 ? dot[g][0] : dot[g][2], O1);
      const float r1 = __shfl_xor_sync(0xffffffffu, up1 ? dot[g][1] : dot[g][3], O1);
      const float a0 = (up1 ? dot[g][2] : dot[g][0]) + r0, a1 = (up1 ? dot[g][3] : dot[g][1]) + r1;
      float s = (up2 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up2 ? a0 : a1, O2);
#pragma unroll
      for (int o = O2 / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s = seen ? s * scale_log2 : -INFINITY;      // log2 domain
      float mx = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, O1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, O2));
      const float m_new = fmaxf(m[g], mx);
      const float m_ref = (m_new == -INFINITY) ? 0.f : m_new;     // a lane group past the end has seen nothing yet
      const float corr = mb::fast_exp2(m[g] - m_ref);             // 2^-inf = 0 on the first step
      prob[g] = mb::fast_exp2(s - m_ref);
      l[g] = l[g] * corr + prob[g];
      m[g] = m_new;
      const mb::f32x2 c2 = mb::pack_f32x2(corr, corr);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[g][i] = mb::mul_f32x2(acc[g][i], c2);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      uint4 raw = make_uint4(0, 0, 0, 0);
      if (live) raw = *reinterpret_cast<const uint4*>(sv + u * PPW * d);
      const mb::f32x2 v0 = mb::bf16x2_to_f32x2(raw.x), v1 = mb::bf16x2_to_f32x2(raw.y),
                      v2 = mb::bf16x2_to_f32x2(raw.z), v3 = mb::bf16x2_to_f32x2(raw.w);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float pu = __shfl_sync(0xffffffffu, prob[g], lane0 | ((u & 2) ? O1 : 0) | ((u & 1) ? O2 : 0));
        const mb::f32x2 p2 = mb::pack_f32x2(pu, pu);
        acc[g][0] = mb::fma_f32x2(p2, v0, acc[g][0]);
        acc[g][1] = mb::fma_f32x2(p2, v1, acc[g][1]);
        acc[g][2] = mb::fma_f32x2(p2, v2, acc[g][2]);
        acc[g][3] = mb::fma_f32x2(p2, v3, acc[g][3]);
      }
    }
  }

  // positions of a warp -> one triple per warp -> one per CTA -> (cluster) one per query head
  __syncthreads();
#pragma unroll
  for (int g = 0; g < G; ++g) {
    l[g] += __shfl_xor_sync(0xffffffffu, l[g], O1);
    l[g] += __shfl_xor_sync(0xffffffffu, l[g], O2);
    float o8[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 t = mb::unpack_f32x2(acc[g][i]);
      o8[2 * i] = t.x;
      o8[2 * i + 1] = t.y;
    }
#pragma unroll
    for (int s = LPP; s < 32; s <<= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m[g], s), lo = __shfl_xor_sync(0xffffffffu, l[g], s);
      const float mn = fmaxf(m[g], mo);
      const float mr = (mn == -INFINITY) ? 0.f : mn;
      const float fa = exp2f(m[g] - mr), fb = exp2f(mo - mr);
      l[g] = l[g] * fa + lo * fb;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float ao = __shfl_xor_sync(0xffffffffu, o8[i], s);
        o8[i] = o8[i] * fa + ao * fb;
      }
      m[g] = mn;
    }
    if (lane == 0) {
      sm.s_m[warp][g] = m[g];
      sm.s_l[warp][g] = l[g];
    }
    if (sub == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) sm.s_acc[warp][g][e0 + i] = o8[i];
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < G * d; t += kWarps * 32) {
    const int g = t / d, e = t - g * d;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, sm.s_m[w][g]);
    const float mr = (M == -INFINITY) ? 0.f : M;
    float L = 0.f, out = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = exp2f(sm.s_m[w][g] - mr);
      L += sm.s_l[w][g] * f;
      out += sm.s_acc[w][g][e] * f;
    }
    if (nsplit == 1) {
      o[(static_cast<long>(b) * nh + h0 + g) * d + e] = __float2bfloat16(L > 0.f ? out / L : 0.f);
    } else {
      sm.c_acc[g][e] = out;
      if (e == 0) {
        sm.c_m[g] = M;
        sm.c_l[g] = L;
      }
    }
  }
  if (nsplit == 1) return;
  sm100::cluster_sync_all();
  // every CTA of the cluster finishes its share of the output elements
  for (int t = split * kWarps * 32 + threadIdx.x; t < G * d; t += nsplit * kWarps * 32) {
    const int g = t / d, e = t - g * d;
    float ms[kMaxSplit], M = -INFINITY;
#pragma unroll
    for (int r = 0; r < kMaxSplit; ++r) {
      ms[r] = r < nsplit ? ld_cluster(&sm.c_m[g], r) : -INFINITY;
      M = fmaxf(M, ms[r]);
    }
    float L = 0.f, out = 0.f;
#pragma unroll
    for (int r = 0; r < kMaxSplit; ++r) {
      if (r < nsplit) {
        const float f = exp2f(ms[r] - M);      // M is finite: position 0 belongs to the first CTA
        L += ld_cluster(&sm.c_l[g], r) * f;
        out += ld_cluster(&sm.c_acc[g][e], r) * f;
      }
    }
    o[(static_cast<long>(b) * nh + h0 + g) * d + e] = __float2bfloat16(L > 0.f ? out / L : 0.f);
  }
  sm100::cluster_sync_all();      // nobody leaves while its shared memory is being read
}

// Short sequences: a CTA per (query head, sequence), a warp per position, loads straight into registers.  What counts
// there is how many CTAs an SM holds and how little one of them costs, not the bytes in flight.
__global__ void __launch_bounds__(kWarps * 32)
decode_attn_short_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, __nv_bfloat16* o,
                         int nh, int group, int d, int len, long q_sb, long k_sb, long k_ss, long k_sh, long v_sb,
                         long v_ss, long v_sh, float scale_log2) {
  const int h = blockIdx.x, b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e0 = lane * 8;
  const bool live = e0 < d;                 // d is a multiple of 8, so a lane is all in or all out
  const int hk = h / group;
  mb::let_next_kernel_start();
  mb::wait_for_previous_kernel();

  float qf[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (live) mb::unpack8(*reinterpret_cast<const mb::bf16x8*>(q + b * q_sb + static_cast<long>(h) * d + e0), qf);
  const __nv_bfloat16* kb = k + b * k_sb + hk * k_sh + e0;
  const __nv_bfloat16* vb = v + b * v_sb + hk * v_sh + e0;

  float m = -INFINITY, l = 0.f;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int j = warp; j < len; j += kWarps) {
    float kf[8], vf[8], dot = 0.f;
    if (live) {
      mb::unpack8(*reinterpret_cast<const mb::bf16x8*>(kb + j * k_ss), kf);
      mb::unpack8(*reinterpret_cast<const mb::bf16x8*>(vb + j * v_ss), vf);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot += qf[i] * kf[i];
    }
    dot = mb::warp_sum(dot) * scale_log2;           // every lane gets the full score (log2 domain)
    const float m_new = fmaxf(m, dot);
    const float m_ref = (m_new == -INFINITY) ? 0.f : m_new;
    const float corr = exp2f(m - m_ref);            // 2^-inf = 0 on the first position
    const float p = exp2f(dot - m_ref);
    l = l * corr + p;
    if (live) {
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = acc[i] * corr + p * vf[i];
    }
    m = m_new;
  }

  __shared__ float s_m[kWarps], s_l[kWarps];
  __shared__ float s_acc[kWarps][kMaxD];
  if (lane == 0) {
    s_m[warp] = m;
    s_l[warp] = l;
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s_acc[warp][e0 + i] = acc[i];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < d; e += kWarps * 32) {
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, s_m[w]);
    const float mr = (M == -INFINITY) ? 0.f : M;
    float L = 0.f, out = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = exp2f(s_m[w] - mr);            // 0 for a warp that saw no position
      L += s_l[w] * f;
      out += s_acc[w][e] * f;
    }
    o[(static_cast<long>(b) * nh + h) * d + e] = __float2bfloat16(L > 0.f ? out / L : 0.f);
  }
}

// Where the short kernel is the faster one; both measured for head sizes 32 - 256, 1 - 96 sequences of 4 - 80 positions
// and one, two and four query heads per CTA of the streaming kernel.  At 12 positions the two meet for one head per CTA.
// More CTAs than are resident at once favour the lighter one for longer (48 x 32 heads of 64: the streaming kernel takes
// 1.54 times as long at 16 positions, 1.01 at 32), and so do few CTAs of four heads, whose steps take four times as long
// (4 x 16 heads of 256 on 4: 1.35 times at 16 positions, 1.14 at 80).
bool short_is_faster(long heads, int group, int d, int len) {
  if (group % 4 == 0) return len <= (heads / 4 > 128 ? 12 : d > 128 ? 96 : 32);
  if (group % 2 == 0) return len <= 16;
  return len <= (heads > 296 ? 40 : 12);
}

// CTAs that share the positions of a (head, sequence): what makes the waves of 296 CTAs (two per SM) cheapest, where a
// CTA costs as much as reading 9600 / d positions (3 us) before its first one and a merge a third of that.  A CTA keeps
// at least 32 positions.  (Doubled up to six waves, 16 x 130 positions of 32 heads of 64 ran as 2048 CTAs of 33 positions.)
int choose_split(long ctas, int len, int d) {
  const long fixed = 9600 / d;
  int best = 1;
  long best_cost = (ctas + 295) / 296 * (fixed + len);
  for (int split = 2; split <= kMaxSplit && len >= 32 * split; split *= 2) {
    const long cost = (ctas * split + 295) / 296 * (fixed + fixed / 3 + (len + split - 1) / split);
    if (cost < best_cost) {
      best_cost = cost;
      best = split;
    }
  }
  return best;
}

template <int LPP, int G, int STAGES>
int launch_decode(const void* q, const void* k, const void* v, void* o, int batch, int nh, int group, int d, int len,
                  long q_sb, long k_sb, long k_ss, long k_sh, long v_sb, long v_ss, long v_sh, float scale_log2,
                  int pdl, cudaStream_t stream) {
  const int split = choose_split(static_cast<long>(batch) * (nh / G), len, d);
  const int chunk = (len + split - 1) / split;
  // stages beyond the ones that a chunk fills would only keep other CTAs away
  const int stage_positions = kWarps * (32 / LPP * kUnroll);
  const int steps = (chunk + stage_positions - 1) / stage_positions;
  const int stages = steps < STAGES ? steps : STAGES;
  const size_t ring = static_cast<size_t>(stages) * stage_positions * 2 * d * 2;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(split, nh / G, batch);
  cfg.blockDim = dim3(kWarps * 32, 1, 1);
  cfg.dynamicSmemBytes = ring > sizeof(MergeArrays<LPP, G>) ? ring : sizeof(MergeArrays<LPP, G>);
  cfg.stream = stream;
  auto kern = decode_attn_kernel<LPP, G, STAGES>;
  static const bool configured =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) == cudaSuccess;
  if (!configured) return -3;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, BF(q), BF(k), BF(v), BFM(o), nh, group, d, len, chunk, stages,
                            q_sb, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, scale_log2) == cudaSuccess
             ? 0
             : -4;
}

// qkv: [tokens][(hq + 2 hk) * d], q heads, then k heads, then v heads.  q is rotated in place; the rotated k and v go
// to rows off + t of the cache ([batch][max_seq][2][hk][d], batch stride `cache_sb`) and nowhere else.  One thread
// per 16 output bytes; the first `rot` channels rotate in halves, cos / sin: [positions][rot / 2] from position `off`.
__global__ void rope_append_kernel(__nv_bfloat16* qkv, __nv_bfloat16* cache,
                                   const float* __restrict__ cosv, const float* __restrict__ sinv, long nvec, int seq,
                                   int hq, int hk, int d, int rot, int off, long cache_sb) {
  const int vpr = (hq + 2 * hk) * (d >> 3);      // 16-byte vectors of one token
  const int vph = d >> 3, half = rot >> 1;
  mb::let_next_kernel_start();
  mb::wait_for_previous_kernel();
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long tok = i / vpr;
    const int w = static_cast<int>(i - tok * vpr);
    const int head = w / vph, c = (w - head * vph) * 8;
    const int t = static_cast<int>(tok % seq);
    const long b = tok / seq;
    __nv_bfloat16* src = qkv + tok * (static_cast<long>(vpr) * 8) + static_cast<long>(head) * d + c;
    const bool rotates = head < hq + hk && c < rot;
    // rotated pairs live in different vectors: the thread of the first half moves both, the other one nothing
    if (rotates && c >= half) continue;
    if (!rotates && head < hq) continue;          // q channels that do not rotate stay where they are
    float x1[8];
    mb::bf16x8 raw = *reinterpret_cast<const mb::bf16x8*>(src);
    __nv_bfloat16* dst = src;
    if (head >= hq) {
      const int which = head >= hq + hk;
      dst = cache + b * cache_sb + (static_cast<long>(off + t) * 2 + which) * hk * d +
            static_cast<long>(head - hq - which * hk) * d + c;
    }
    if (rotates) {
      float x2[8], o1[8], o2[8];
      mb::unpack8(raw, x1);
      mb::unpack8(*reinterpret_cast<const mb::bf16x8*>(src + half), x2);
      const float* cs = cosv + static_cast<long>(t) * half + c;
      const float* sn = sinv + static_cast<long>(t) * half + c;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        o1[e] = x1[e] * cs[e] - x2[e] * sn[e];
        o2[e] = x1[e] * sn[e] + x2[e] * cs[e];
      }
      *reinterpret_cast<mb::bf16x8*>(dst) = mb::pack8(o1);
      *reinterpret_cast<mb::bf16x8*>(dst + half) = mb::pack8(o2);
    } else {
      *reinterpret_cast<mb::bf16x8*>(dst) = raw;
    }
  }
}

}  // namespace

// q: [batch][nh][d] with batch stride q_sb; o: contiguous, bf16.  k, v: element strides (batch, position, kv head)
// with unit stride along d; every row start must be 16-byte aligned (strides multiples of 8).  d % 8 == 0,
// d <= 256, nh % nh_kv == 0, len >= 1.  pdl: launch as a dependent of the kernel before (see the fetch order above:
// only position len - 1 of the cache may have been written by that kernel).
MB_API int mb_decode_attn(const void* q, const void* k, const void* v, void* o, int batch, int nh, int nh_kv, int d,
                          int len, long q_sb, long k_sb, long k_ss, long k_sh, long v_sb, long v_ss, long v_sh,
                          float scale, int pdl, cudaStream_t stream) {
  if (batch <= 0 || nh <= 0) return 0;
  if (d % 8 || d > kMaxD || d <= 0 || nh_kv <= 0 || nh % nh_kv || len < 1) return -1;
  if ((q_sb | k_sb | k_ss | k_sh | v_sb | v_ss | v_sh) & 7) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15)
    return -1;
  const int group = nh / nh_kv;
  const float sl = scale * 1.4426950408889634f;
#define MB_DECODE(L_, G_, S_)                                                                                        \
  return launch_decode<L_, G_, S_>(q, k, v, o, batch, nh, group, d, len, q_sb, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, sl, \
                                   pdl, stream)
#define MB_DECODE_G(L_, S_)                   \
  do {                                        \
    if (group % 4 == 0) MB_DECODE(L_, 4, S_); \
    if (group % 2 == 0) MB_DECODE(L_, 2, S_); \
    MB_DECODE(L_, 1, S_);                     \
  } while (0)
  if (short_is_faster(static_cast<long>(batch) * nh, group, d, len)) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(nh, batch, 1);
    cfg.blockDim = dim3(kWarps * 32, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, decode_attn_short_kernel, BF(q), BF(k), BF(v), BFM(o), nh, group, d, len, q_sb,
                              k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, sl) == cudaSuccess
               ? 0
               : -4;
  }
  // stages per warp: four where two CTAs of them fit an SM, else three (up to 96 KB per CTA)
  if (d <= 48) MB_DECODE_G(8, 4);
  if (d <= 64) MB_DECODE_G(8, 3);
  if (d <= 96) MB_DECODE_G(16, 4);
  if (d <= 128) MB_DECODE_G(16, 3);
  MB_DECODE_G(32, 3);
#undef MB_DECODE_G
#undef MB_DECODE
}

// See rope_append_kernel.  rot % 16 == 0 (0: no rotation, cos / sin unused), d % 8 == 0, qkv and cache 16-byte aligned.
MB_API int mb_rope_append(void* qkv, void* cache, const float* cosv, const float* sinv, int batch, int seq, int hq,
                          int hk, int d, int rot, int off, long cache_sb, int pdl, cudaStream_t stream) {
  if (rot % 16 || rot > d || d % 8 || cache_sb % 8) return -1;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(cache)) & 15) return -1;
  const long nvec = static_cast<long>(batch) * seq * (hq + 2 * hk) * (d / 8);
  if (!nvec) return 0;
  long blocks = (nvec + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(static_cast<unsigned>(blocks), 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, rope_append_kernel, BFM(qkv), BFM(cache), cosv, sinv, nvec, seq, hq, hk, d, rot, off,
                            cache_sb) == cudaSuccess
             ? 0
             : -4;
}
