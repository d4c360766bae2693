// Attention forward with two 128-row query tiles per CTA; included by attn_fwd_tcgen05.cu, which chooses between
// this kernel and the one-tile kernel.
//
// What bounds attention at head size 128 is the exponential unit and the tensor pipe alike (about 1024 cycles
// each per 128 x 128 block), so both have to run all the time.  One CTA per SM therefore keeps two query tiles
// in flight: while one tile's exponentials are computed, the other tile's products run.  One MMA warp serves the
// tiles in turn; with a warp for each, their products interleaved and both tiles' scores arrived together.
// A tile has two warpgroups, each with 64 of the 128 keys of a block (one row per thread, the row maximum goes
// through shared memory): with one warpgroup and 128 keys a thread, a scheduler had one warp to issue from, and a
// block took 2690 cycles per tile instead of XXX.
// P never leaves tensor memory: it overwrites S columns of its own half and is the A operand of the P V product.
// Per tile the order is S(j), softmax, P V(j), S(j+1); P V(j) and S(j+1) are issued back to back, in order, so
// S(j+1) may overwrite P(j), and the arrival of S(j+1) tells the softmax warps that P V(j) is done, which is when O
// may be rescaled.
//
// The grid is persistent, one CTA per SM.  The work list is ordered by groups of heads whose keys and values fit
// L2 together, inside a group by query tile, those with most blocks (causal mask) first, and dealt forwards and
// backwards in turn, so the CTAs end together.
//
// Tensor memory: S0 at column 0, S1 at 128, O0 at 256, O1 at 384; P of keys 64 h ... at S + 64 h.
// Warps 0-7: softmax and output of tile 0; 8-15: tile 1; 16: K / V loads; 17: MMA; 18: Q loads.
#pragma once

namespace duo {

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

__device__ __forceinline__ void store32(__nv_bfloat16* dst, const float* f, bool wide) {
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
attn_fwd_duo_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const AttnParams p, const Sched sch) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + oBar);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 2;
  uint64_t* full = bars + 4;
  uint64_t* empty = full + kSlots;
  uint64_t* s_full = empty + kSlots;
  uint64_t* p_full = s_full + 2;            // [tile][half of the keys]
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
      mbar_init(&p_full[2 * i], 4);           // one arrival of each warp of the half
      mbar_init(&p_full[2 * i + 1], 4);
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
      int n = 0, cq[2] = {0, 0}, cp[2] = {0, 0};   // ring position, Q tiles and P tiles so far
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
      // S(j) = Q K(j)^T of tile i from ring position at; tile 1 comes last and releases the slot
      auto key_step = [&](const Work& w, int i, int j, int at) {
        const int active = i ? w.nb[1] : w.nb[0];
        const int slot = at % kSlots;
        if (j == 0 && active > 0) {
          if (!wait(&q_full[i], cq[i], MB_ERR_TIMEOUT_FULL)) return;
          ++cq[i];
        }
        if (!wait(&full[slot], at / kSlots, MB_ERR_TIMEOUT_FULL)) return;
        tc_fence_after();
        if (elect_one()) {
          if (j < active) {
            const uint64_t dq = make_smem_desc_sw128(base + i * kTile, 16, 1024);
            const uint64_t dk = make_smem_desc_sw128(base + oRing + slot * kTile, 16, 1024);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              const uint32_t off = ((kk >> 2) * kChunk + (kk & 3) * 32) >> 4;
              if (kk < ksteps) mma_f16_ss(tmem_base + i * 128, dq + off, dk + off, idesc_s, kk != 0 ? 1u : 0u);
            }
            mma_commit(&s_full[i]);
            if (j == active - 1) mma_commit(&q_empty[i]);
          }
          if (i == 1) mma_commit(&empty[slot]);
        }
        __syncwarp();
      };
      Work cur = next_work();
      for (int i = 0; i < 2 && cur.nbmax > 0; ++i) key_step(cur, i, 0, 0);
      while (ok && cur.nbmax > 0) {
        const Work nxt = next_work();
        for (int j = 0; j < cur.nbmax && ok; ++j, n += 2) {
          const int slot = (n + 1) % kSlots;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int active = cur.nb[i];
            if (!wait(&full[slot], (n + 1) / kSlots, MB_ERR_TIMEOUT_FULL)) break;
            if (j < active) {
              const uint32_t t_s = tmem_base + i * 128, t_o = tmem_base + 256 + i * 128;
              // V: [keys][64-wide d atoms], 16 keys = 2048 B
              const uint64_t dv = make_smem_desc_sw128(base + oRing + slot * kTile, kChunk, 1024);
              // the first product of an item overwrites O: both halves have to have read the last item's
              if (j == 0 && !wait(&p_full[2 * i + 1], cp[i], MB_ERR_TIMEOUT_TMEM)) break;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                if (!wait(&p_full[2 * i + h], cp[i], MB_ERR_TIMEOUT_TMEM)) break;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int kk = 4 * h; kk < 4 * h + 4; ++kk)       // 16 keys of P are 8 columns
                    mma_f16_ts(t_o, t_s + 64 * h + 8 * (kk & 3), dv + kk * (2048 >> 4), idesc_o,
                               (j | kk) != 0 ? 1u : 0u);
                  if (h == 1 && j == active - 1) mma_commit(&o_full[i]);
                }
                __syncwarp();
              }
              if (!ok) break;
              ++cp[i];
            }
            if (i == 1 && elect_one()) mma_commit(&empty[slot]);
            __syncwarp();
            if (j + 1 < cur.nbmax) key_step(cur, i, j + 1, n + 2);
            else if (nxt.nbmax > 0) key_step(nxt, i, 0, n + 2);
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
        if (__any_sync(0xffffffffu, j > 0 && alpha != 1.f)) {      // the same in both warps of the pair
          for (int c = 16 * h; c < p.d_mma; c += 32) {
            uint32_t o[16];
            tmem_ld16(t_o + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int u = 0; u < 16; ++u) o[u] = __float_as_uint(__uint_as_float(o[u]) * alpha);
            tmem_st16(t_o + c, o);
          }
          tmem_st_wait();
          tc_fence_before();
          pair_sync();
          tc_fence_after();
        }
        const mb::f32x2 m2 = mb::pack_f32x2(m_neg, m_neg);
        mb::f32x2 sum0 = 0, sum1 = 0;
        uint32_t pk[32];
#pragma unroll
        for (int c = 0; c < 64; c += 4) {
          const uint32_t* s4 = sr + c;
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
        tmem_st32(t_s, pk);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(&p_full[2 * i + h]);
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
          store32(orow + c, f, wide);
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

}  // namespace duo
