// Causal / full multi-head attention forward on tcgen05 tensor cores.
//
//   O = softmax(scale * Q K^T + causal mask) V,   LSE = logsumexp per row
//
// What bounds attention at head size 128 is the exponential unit and the tensor pipe alike (about 1024 cycles
// each per 128 x 128 block), so both have to run all the time.  One CTA per SM therefore keeps two query tiles
// in flight: while one tile's exponentials are computed, the other tile's products run.  One MMA warp serves the
// tiles in turn; with a warp for each, their products interleaved and both tiles' scores arrived together.
// A tile has two warpgroups, each with 64 of the 128 keys of a block (one row per thread, the row maximum goes
// through shared memory), so that a scheduler has two warps of a tile to issue from.
// P never leaves tensor memory: it overwrites S columns of its own half and is the A operand of the P V product.
// Per tile the order is S(j), softmax, P V(j), S(j+1); P V(j) and S(j+1) are issued back to back, in order, so
// S(j+1) may overwrite P(j), and the arrival of S(j+1) tells the softmax warps that P V(j) is done, which is when O
// may be rescaled.  P is handed over in two parts, so half of its product hides behind the other half's exponentials.
// Measured (cycles): a tile's softmax 2000, its products 1250 with the waits between them, a period of 3400 for both
// tiles; 32 heads of 128, 8192 tokens, no mask: 1145 -> 961 us (1144 TFLOP/s); 8 x 2048 tokens, 32 heads of 80,
// causal: 391 -> 257 us; 2 x 256 tokens, 4 heads of 128, causal: 11.2 -> 9.8 us.  The left sides are the kernel
// before: one tile per CTA, two CTAs per SM, 64 keys per block, P through shared memory.
//
// The grid is persistent, one CTA per SM.  The work list is ordered by groups of heads whose keys and values fit
// L2 together, inside a group by query tile, those with most blocks (causal mask) first, and dealt forwards and
// backwards in turn, so the CTAs end together.
//
// Tensor memory: S0 at column 0, S1 at 128, O0 at 256, O1 at 384; P of keys 64 h ... at S + 64 h.
// Warps 0-7: softmax and output of tile 0; 8-15: tile 1; 16: K / V loads; 17: MMA; 18: Q loads.
//
// Q, K and V tiles arrive by per-CTA TMA (4-D tensor maps over [batch][token][head][d], so a packed qkv projection
// output is consumed in place; head sizes that are not a multiple of 64, e.g. 80, are zero-filled by the TMA bounds
// check instead of being padded in memory).
//
// Replaces the reference's flash-attention v2 forward, an sm_80 mma.sync kernel
// (reference: csrc/flash_attn/src/flash_fwd_kernel.h, flash_fwd_launch_template.h:13-28,
// dispatch mist/modules/flash_attn.py:46-213).
#include "sm100.cuh"

using namespace sm100;

namespace {

constexpr int BM = 128;
constexpr int BN = 128;
constexpr int kThreads = 640;
constexpr int kSlots = 5;                 // ring of K and V tiles in the order K0 V0 K1 V1 ...
constexpr int kTile = 2 * 128 * 128;      // 128 rows of up to two 64-wide chunks
constexpr int oRing = 2 * kTile;
constexpr int oBar = oRing + kSlots * kTile;
// q_full[2], q_empty[2], full[5], empty[5], s_full[2], p_full[2][2], o_full[2]
constexpr int kNumBars = 2 + 2 + kSlots + kSlots + 2 + 4 + 2;
constexpr int oMax = oBar + kNumBars * 8 + 16;      // [tile][half][row] maxima (and, at the end, sums)
constexpr int kSmem = oMax + 2 * 2 * BM * 4;
static_assert(kSmem <= 232448, "attention forward: shared memory over the per-CTA limit");

struct AttnParams {
  __nv_bfloat16* o;
  float* lse;
  int sq, sk, nh, nh_kv, d, d_mma, nchunks;
  long o_batch_stride, o_tok_stride, o_head_stride;
  float scale_log2;
  int causal;
  // per-sample lengths of a right-padded batch (null: every sample has sq / sk tokens): queries and keys
  // at or past a sample's length are padding -- such keys are masked, such query rows come out as zeros
  const int* seqlens_q;
  const int* seqlens_k;
  int* status;
};

__device__ __forceinline__ void report(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}

struct Sched {
  int npairs;      // pairs of query tiles per (batch, head)
  int bh;          // batch * heads
  int group;       // (batch, head)s that are walked together
  int total;
};

struct Work {
  int q0[2], nb[2], nbmax, head, batch, sq_b, sk_b, coff;
};

__device__ __forceinline__ int work_index(int n) {
  const int c = (n & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  return n * gridDim.x + c;
}

__device__ __forceinline__ Work work_at(const AttnParams& p, const Sched& s, int t) {
  Work w;
  const int per_group = s.group * s.npairs;
  const int g = t / per_group, r = t - g * per_group;
  const int gsize = min(s.group, s.bh - g * s.group);
  const int qi = r / gsize;
  const int bh = g * s.group + (r - qi * gsize);
  w.batch = bh / p.nh;
  w.head = bh - w.batch * p.nh;
  w.sq_b = p.seqlens_q ? min(p.sq, p.seqlens_q[w.batch]) : p.sq;
  w.sk_b = p.seqlens_k ? min(p.sk, p.seqlens_k[w.batch]) : p.sk;
  w.coff = w.sk_b - w.sq_b;
  w.nbmax = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int q0 = (2 * (s.npairs - 1 - qi) + i) * BM;
    int nb = (q0 < w.sq_b) ? (w.sk_b + BN - 1) / BN : 0;
    if (p.causal) {
      const int last = q0 + BM - 1 + w.coff;
      nb = min(nb, last < 0 ? 0 : last / BN + 1);
    }
    w.q0[i] = q0;
    w.nb[i] = nb;
    w.nbmax = max(w.nbmax, nb);
  }
  return w;
}

__device__ __forceinline__ void store16(__nv_bfloat16* dst, const float* f, bool wide) {
  const mb::bf16x8 a = mb::pack8(f), b = mb::pack8(f + 8);
  if (wide) {
    const uint32_t* x = reinterpret_cast<const uint32_t*>(&a);
    const uint32_t* y = reinterpret_cast<const uint32_t*>(&b);
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(dst), "r"(x[0]), "r"(x[1]),
                 "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3])
                 : "memory");
  } else {
    reinterpret_cast<mb::bf16x8*>(dst)[0] = a;
    reinterpret_cast<mb::bf16x8*>(dst)[1] = b;
  }
}

__global__ void __launch_bounds__(kThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const AttnParams p, const Sched sch) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + oBar);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 2;
  uint64_t* full = bars + 4;
  uint64_t* empty = full + kSlots;
  uint64_t* s_full = empty + kSlots;
  uint64_t* p_full = s_full + 2;            // [tile][first, second 32 keys of each half]
  uint64_t* o_full = p_full + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled tiles need a 1024-byte base
    if (threadIdx.x == 0) report(p.status, MB_ERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&o_full[i], 1);
      mbar_init(&p_full[2 * i], 8);           // one arrival of each warp of the tile
      mbar_init(&p_full[2 * i + 1], 8);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    fence_barrier_init();
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
  }
  if (warp == 16) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  constexpr uint32_t kChunk = 128 * 128;

  if (warp >= 16) {
    // 640 threads were launched with 96 registers; 512 * 104 + 128 * 64 is the same sum
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;\n");
    if (warp == 16) {
      // ---------------------------------------------------------- K, V producer
      if (lane == 0) {
        int n = 0, slot = 0;
        bool ok = true;
        auto load = [&](const CUtensorMap* tm, int row, int head_kv, int batch) {
          if (n >= kSlots && !mbar_wait(&empty[slot], (n / kSlots - 1) & 1)) {
            report(p.status, MB_ERR_TIMEOUT_EMPTY);
            ok = false;
            return;
          }
          uint8_t* dst = smem + oRing + slot * kTile;
          mbar_expect_tx(&full[slot], p.nchunks * kChunk);
          for (int c = 0; c < p.nchunks; ++c)
            tma_load_4d(dst + c * kChunk, tm, &full[slot], 64 * c, head_kv, row, batch);
          ++n;
          if (++slot == kSlots) slot = 0;
        };
        for (int r = 0; ok; ++r) {
          const int t = work_index(r);
          if (t >= sch.total) break;
          const Work w = work_at(p, sch, t);
          const int head_kv = w.head / (p.nh / p.nh_kv);
          for (int j = 0; j < w.nbmax && ok; ++j) {
            load(&tm_k, j * BN, head_kv, w.batch);
            if (ok) load(&tm_v, j * BN, head_kv, w.batch);
          }
        }
      }
    } else if (warp == 18) {
      // ------------------------------------------------------------- Q producer
      if (lane == 0) {
        int cq[2] = {0, 0};
        bool ok = true;
        for (int r = 0; ok; ++r) {
          const int t = work_index(r);
          if (t >= sch.total) break;
          const Work w = work_at(p, sch, t);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (w.nb[i] == 0 || !ok) continue;
            if (cq[i] > 0 && !mbar_wait(&q_empty[i], (cq[i] - 1) & 1)) {
              report(p.status, MB_ERR_TIMEOUT_EMPTY);
              ok = false;
              continue;
            }
            mbar_expect_tx(&q_full[i], p.nchunks * kChunk);
            for (int c = 0; c < p.nchunks; ++c)
              tma_load_4d(smem + i * kTile + c * kChunk, &tm_q, &q_full[i], 64 * c, w.head, w.q0[i], w.batch);
            ++cq[i];
          }
        }
      }
    } else if (warp == 17) {
      // ------------------------------------------------------------- MMA issuer
      const uint32_t idesc_s = make_idesc_bf16(BM, BN, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(BM, p.d_mma, 0, 1);
      const uint32_t base = smem_u32(smem);
      const int ksteps = p.d_mma / 16;
      int cq[2] = {0, 0}, cp[2] = {0, 0};    // Q tiles and P tiles so far
      int round = 0;
      bool ok = true;
      auto wait = [&](uint64_t* bar, int phase, int code) -> bool {
        if (ok && !mbar_wait(bar, phase & 1)) {
          report(p.status, code);
          ok = false;
        }
        return ok;
      };
      // The next item of the list with a block to compute; nbmax = 0 at the end of the list.
      auto next_work = [&]() -> Work {
        for (;;) {
          const int t = work_index(round++);
          Work w;
          w.nbmax = 0;
          if (t < sch.total) w = work_at(p, sch, t);
          if (t >= sch.total || w.nbmax > 0) return w;
        }
      };
      // Next slot of the ring, once it is full.
      int slot = 0, lap = 0;
      auto take_slot = [&]() -> int {
        const int at = slot;
        wait(&full[at], lap, MB_ERR_TIMEOUT_FULL);
        if (++slot == kSlots) { slot = 0; lap ^= 1; }
        return at;
      };
      // S(j) = Q K(j)^T of tile i; tile 1 comes last and releases the slot
      auto issue_s = [&](int i, int at, bool active, bool last) {
        if (elect_one()) {
          if (active) {
            const uint64_t dq = make_smem_desc_sw128(base + i * kTile, 16, 1024);
            const uint64_t dk = make_smem_desc_sw128(base + oRing + at * kTile, 16, 1024);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              const uint32_t off = ((kk >> 2) * kChunk + (kk & 3) * 32) >> 4;
              if (kk < ksteps) mma_f16_ss(tmem_base + i * 128, dq + off, dk + off, idesc_s, kk != 0 ? 1u : 0u);
            }
            mma_commit(&s_full[i]);
            if (last) mma_commit(&q_empty[i]);
          }
          if (i == 1) mma_commit(&empty[at]);
        }
        __syncwarp();
      };
      // the first S of an item also waits for its Q tile
      auto first_s = [&](const Work& w, int i, int at) {
        if (w.nb[i] > 0) wait(&q_full[i], cq[i]++, MB_ERR_TIMEOUT_FULL);
        if (!ok) return;
        tc_fence_after();
        issue_s(i, at, w.nb[i] > 0, w.nb[i] == 1);
      };
      Work cur = next_work();
      if (cur.nbmax > 0) {
        const int at = take_slot();
        first_s(cur, 0, at);
        first_s(cur, 1, at);
      }
      while (ok && cur.nbmax > 0) {
        const Work nxt = next_work();
        for (int j = 0; j < cur.nbmax && ok; ++j) {
          const bool inside = j + 1 < cur.nbmax;
          const int at_v = take_slot();
          int at_k = 0;
          if (inside || nxt.nbmax > 0) at_k = take_slot();
          if (!ok) break;
          const uint64_t dv = make_smem_desc_sw128(base + oRing + at_v * kTile, kChunk, 1024);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int active = cur.nb[i];
            if (j < active) {
              const uint32_t t_s = tmem_base + i * 128, t_o = tmem_base + 256 + i * 128;
#pragma unroll
              for (int part = 0; part < 2; ++part) {
                if (!wait(&p_full[2 * i + part], cp[i], MB_ERR_TIMEOUT_TMEM)) break;
                tc_fence_after();
                if (elect_one()) {
                  // part 0: the first 32 keys of both halves; 16 keys are 8 columns of P and 2048 B of V
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    const int kk = 4 * (u >> 1) + 2 * part + (u & 1);
                    mma_f16_ts(t_o, t_s + 64 * (kk >> 2) + 8 * (kk & 3), dv + kk * (2048 >> 4), idesc_o,
                               (j | kk) != 0 ? 1u : 0u);
                  }
                  if (part == 1 && j == active - 1) mma_commit(&o_full[i]);
                }
                __syncwarp();
              }
              if (!ok) break;
              ++cp[i];
            }
            if (i == 1 && elect_one()) mma_commit(&empty[at_v]);
            __syncwarp();
            if (inside) issue_s(i, at_k, j + 1 < active, j + 2 == active);
            else if (nxt.nbmax > 0) first_s(nxt, i, at_k);
          }
        }
        cur = nxt;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;\n");
    // ------------------------------------------------------- softmax and output
    const int i = warp >> 3;          // query tile
    const int h = (warp >> 2) & 1;    // half of the keys of a block, and of the output's columns
    const int r = threadIdx.x & 127;  // row of the tile == TMEM lane
    const int pair_bar = 1 + 4 * i + (warp & 3);      // named barrier of the two warps that share these rows
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem_base + i * 128 + 64 * h + lane_off, t_o = tmem_base + 256 + i * 128 + lane_off;
    float* s_max = reinterpret_cast<float*>(smem + oMax) + i * 2 * BM + r;    // [half]
    const mb::f32x2 scale2 = mb::pack_f32x2(p.scale_log2, p.scale_log2);
    const bool wide = ((reinterpret_cast<uintptr_t>(p.o) & 31) | ((p.o_tok_stride | p.o_head_stride |
                       p.o_batch_stride) & 15)) == 0;
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory"); };
    int cs = 0, co = 0;               // S tiles and O tiles so far
    bool ok = true;
    for (int rnd = 0; ok; ++rnd) {
      const int t = work_index(rnd);
      if (t >= sch.total) break;
      const Work w = work_at(p, sch, t);
      const int q0 = i ? w.q0[1] : w.q0[0], nb = i ? w.nb[1] : w.nb[0];
      const int qi = q0 + r;
      const int vis = (p.causal ? min(w.sk_b - 1, qi + w.coff) : w.sk_b - 1) - 64 * h;   // last visible key of the row
      const int vis_tile = p.causal ? min(w.sk_b - 1, q0 + w.coff) : w.sk_b - 1;         // of the tile's first row
      float m_run = -INFINITY, l_run = 0.f;

      for (int j = 0; j < nb; ++j) {
        if (!mbar_wait(&s_full[i], cs & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t sr[64];
        tmem_ld32(t_s, sr);
        tmem_ld32(t_s + 32, sr + 32);
        tmem_ld_wait();
        if (j * BN + BN - 1 > vis_tile) {
          const int lim = vis - j * BN;      // last visible column
#pragma unroll
          for (int c = 0; c < 64; ++c) sr[c] = (c <= lim) ? sr[c] : 0xff800000u;
        }
        float mx[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) mx[u] = fmaxf(__uint_as_float(sr[u]), __uint_as_float(sr[4 + u]));
#pragma unroll
        for (int c = 8; c < 64; c += 8) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            mx[u] = fmaxf(mx[u], fmaxf(__uint_as_float(sr[c + u]), __uint_as_float(sr[c + 4 + u])));
        }
        // the next write comes after the next s_full, that is after the other half's arrival on p_full, below its read
        const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        s_max[h * BM] = mine;
        pair_sync();
        ++cs;
        // raw scores; the softmax scale (> 0, so maxima commute with it) is folded into the FFMA below
        const float mxs = fmaxf(mine, s_max[(h ^ 1) * BM]) * p.scale_log2;
        // Lazy rescaling: keep the old reference maximum unless the new one is much larger; probabilities then
        // stay below 2^8, harmless in fp32 / bf16.
        const float m_new = fmaxf(m_run, mxs);
        const float m_use = (m_new - m_run > 8.f || m_run == -INFINITY) ? m_new : m_run;
        const float alpha = (m_run == -INFINITY) ? 0.f : exp2f(m_run - m_use);
        const float m_neg = (m_use == -INFINITY) ? 0.f : -m_use;
        // S(j) is complete, so P V(j-1), issued before it, is too: O may be rescaled, each half its columns
        if (__any_sync(0xffffffffu, j > 0 && alpha != 1.f)) {      // before the arrivals on p_full, which P V waits for
          for (int c = 16 * h; c < p.d_mma; c += 32) {
            uint32_t o[16];
            tmem_ld16(t_o + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int u = 0; u < 16; ++u) o[u] = __float_as_uint(__uint_as_float(o[u]) * alpha);
            tmem_st16(t_o + c, o);
          }
        }
        const mb::f32x2 m2 = mb::pack_f32x2(m_neg, m_neg);
        mb::f32x2 sum0 = 0, sum1 = 0;
        // P in two parts, so that the first half of its product runs beside the second half of the exponentials
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          uint32_t pk[16];
#pragma unroll
          for (int c = 0; c < 32; c += 4) {
            const uint32_t* s4 = sr + 32 * part + c;
            const float2 xa = mb::unpack_f32x2(
                mb::fma_f32x2(mb::pack_f32x2(__uint_as_float(s4[0]), __uint_as_float(s4[1])), scale2, m2));
            const float2 xb = mb::unpack_f32x2(
                mb::fma_f32x2(mb::pack_f32x2(__uint_as_float(s4[2]), __uint_as_float(s4[3])), scale2, m2));
            const float a0 = mb::fast_exp2(xa.x), a1 = mb::fast_exp2(xa.y);
            const float b0 = mb::fast_exp2(xb.x), b1 = mb::fast_exp2(xb.y);
            sum0 = mb::add_f32x2(sum0, mb::pack_f32x2(a0, a1));
            sum1 = mb::add_f32x2(sum1, mb::pack_f32x2(b0, b1));
            pk[c >> 1] = pack_bf16x2(a0, a1);
            pk[(c >> 1) + 1] = pack_bf16x2(b0, b1);
          }
          tmem_st16(t_s + 16 * part, pk);
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive_warp(&p_full[2 * i + part]);
        }
        const float2 sum = mb::unpack_f32x2(mb::add_f32x2(sum0, sum1));
        l_run = l_run * alpha + (sum.x + sum.y);
        m_run = m_use;
      }
      if (!ok) break;

      if (nb > 0) {
        if (!mbar_wait(&o_full[i], co & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        ++co;
        tc_fence_after();
      }
      // the other half's share of the row sum (the last block's P V is done: both halves have read the maxima)
      s_max[h * BM] = l_run;
      pair_sync();
      l_run = s_max[0] + s_max[BM];
      pair_sync();
      const bool real_row = qi < w.sq_b;
      const float inv = (real_row && l_run > 0.f) ? 1.f / l_run : 0.f;
      __nv_bfloat16* orow = p.o + w.batch * p.o_batch_stride + static_cast<long>(qi) * p.o_tok_stride +
                            static_cast<long>(w.head) * p.o_head_stride;
      for (int c = 16 * h; c < p.d; c += 32) {
        uint32_t o[16];
        if (nb > 0) {
          tmem_ld16(t_o + c, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int u = 0; u < 16; ++u) o[u] = 0;
        }
        if (qi < p.sq) {
          float f[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) f[u] = __uint_as_float(o[u]) * inv;
          store16(orow + c, f, wide);
        }
      }
      tc_fence_before();
      if (h == 0 && qi < p.sq)
        p.lse[(static_cast<long>(w.batch) * p.nh + w.head) * p.sq + qi] =
            (real_row && l_run > 0.f) ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 16) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

#include "attn_fwd_one_tile_tcgen05.cuh"

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) !=
            cudaSuccess || q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// [batch][tokens][heads][d] bf16 with element strides; box = [1][rows][1][64].
bool make_map(CUtensorMap* m, const void* base, int batch, int tokens, int heads, int d,
              long batch_stride, long tok_stride, long head_stride, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(heads),
                        static_cast<cuuint64_t>(tokens), static_cast<cuuint64_t>(batch)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(head_stride) * 2,
                           static_cast<cuuint64_t>(tok_stride) * 2,
                           static_cast<cuuint64_t>(batch_stride) * 2};
  cuuint32_t box[4] = {64, 1, static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_with_context([&] {
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}

}  // namespace

MB_API int* mb_status_device_ptr();

// q: [batch][sq][nh][d], k/v: [batch][sk][nh_kv][d], element strides given per tensor
// (so views into a packed qkv buffer work).  o: [batch][sq][nh][d] with its own strides.
// lse: [batch][nh][sq] fp32.  Head size d: multiple of 16, <= 128; all strides
// multiples of 8 elements and base pointers 16-byte aligned.  seqlens_q / seqlens_k: optional device
// arrays of `batch` ints, the number of real tokens of each sample of a right-padded batch (what the
// reference handles by removing the padding and calling its variable-length kernels,
// csrc/flash_attn/flash_api.cpp:427); padded query rows get zeros and lse = -inf.
MB_API int mb_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int batch,
                       int sq, int sk, int nh, int nh_kv, int d, long q_bs, long q_ts, long q_hs,
                       long k_bs, long k_ts, long k_hs, long v_bs, long v_ts, long v_hs, long o_bs,
                       long o_ts, long o_hs, float scale, int causal, const int* seqlens_q,
                       const int* seqlens_k, cudaStream_t stream) {
  if (d % 16 || d > 128 || d < 16 || nh % nh_kv) return -1;
  if ((q_ts | q_hs | q_bs | k_ts | k_hs | k_bs | v_ts | v_hs | v_bs | o_ts | o_hs | o_bs) & 7) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
       reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(o)) & 15)
    return -1;
  if (batch == 0 || sq == 0) return 0;
  const long pairs = (sq + 2 * BM - 1) / (2 * BM), units = pairs * nh * batch;
  if (units > 0x3fffffff) return -1;
  CUtensorMap tq, tk, tv;
  if (!make_map(&tq, q, batch, sq, nh, d, q_bs, q_ts, q_hs, BM)) return -2;
  const bool small = one_tile::is_faster(sq, sk, static_cast<long>(nh) * batch, d) && nh <= 65535 && batch <= 65535;
  const int bn = small ? one_tile::BN : BN;
  if (!make_map(&tk, k, batch, sk, nh_kv, d, k_bs, k_ts, k_hs, bn)) return -2;
  if (!make_map(&tv, v, batch, sk, nh_kv, d, v_bs, v_ts, v_hs, bn)) return -2;
  AttnParams p;
  p.o = reinterpret_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.sq = sq; p.sk = sk; p.nh = nh; p.nh_kv = nh_kv; p.d = d;
  p.d_mma = d;
  p.nchunks = (d + 63) / 64;
  p.o_batch_stride = o_bs; p.o_tok_stride = o_ts; p.o_head_stride = o_hs;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.seqlens_q = seqlens_q;
  p.seqlens_k = seqlens_k;
  p.status = mb_status_device_ptr();
  if (small) {
    static bool cfg = false;
    if (!cfg) {
      if (cudaFuncSetAttribute(one_tile::attn_fwd_one_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               one_tile::Smem::kTotal) != cudaSuccess)
        return -3;
      cfg = true;
    }
    one_tile::attn_fwd_one_tile_kernel<<<dim3((sq + BM - 1) / BM, nh, batch), one_tile::kThreads,
                                         one_tile::Smem::kTotal, stream>>>(tq, tk, tv, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -4;
  }
  static bool cfg = false;
  if (!cfg) {
    if (cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess)
      return -3;
    cfg = true;
  }
  Sched sch;
  sch.npairs = static_cast<int>(pairs);
  sch.bh = nh * batch;
  // heads whose keys and values take about a third of L2 together, at least one key / value head
  const long kv_bytes = 4l * sk * d;
  const long kv_heads = kv_bytes > 0 ? (40l << 20) / kv_bytes : 1;
  const long group = (kv_heads < 1 ? 1 : kv_heads) * (nh / nh_kv);
  sch.group = static_cast<int>(group < sch.bh ? group : sch.bh);
  sch.total = static_cast<int>(units);
  attn_fwd_kernel<<<units < 148 ? static_cast<int>(units) : 148, kThreads, kSmem, stream>>>(tq, tk, tv, p, sch);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
