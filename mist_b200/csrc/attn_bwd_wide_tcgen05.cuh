// Attention backward on 128 x 128 blocks; included by attn_bwd_tcgen05.cu.
//
// A CTA owns a 128-row key/value block of one key/value head (or of some of its query heads) and walks the query
// blocks of its query heads; dV and dK stay in tensor memory all the while.  Rows of every score tile are keys:
//
//   S^T  = K Q^T      P^T = exp2(S^T*c - LSE)      dV += P^T dO    (A = P^T in tensor memory, over S^T)
//   dP^T = V dO^T     dS^T = P^T o (dP^T - delta)  dK += dS^T Q    (A = dS^T in shared memory)
//                                                  dQ  = dS K      (A = the same tile read MN-major)
//
// The softmax scale multiplies dK once at the end and dQ in the conversion to bf16, in fp32.
// What bounds a block: five products of 512 cycles each at head size 128, and shared memory, which feeds them at
// 128 B a cycle.  128 query rows per block instead of 64 are what makes the two meet: a 128 x 64 product takes its
// operands from shared memory at two thirds of the tensor rate.  The MMA warp issues S^T of block i+1 before it
// waits for dS^T of block i, so the exponentials run beside the dQ, dK products of the block before.
// dQ is added to an fp32 accumulator with TMA reduces by a warpgroup of its own: about 850 cycles per 128 x 32 values,
// which at head size 128 is as long as the block's products.  (Untiled bulk reduces of the same bytes into a contiguous
// accumulator took 1150.)
//
// Tensor memory (columns): head size up to 80: S^T 0, dP^T 128, dQ 256, dV 336, dK 416; above, dQ has no columns of
// its own and takes dP^T's: S^T 0, dP^T / dQ 128, dV 256, dK 384.
//
// Persistent, one CTA per SM; the work list is ordered by groups of heads whose tensors share L2 and inside a group
// by key block (under the causal mask the first blocks are the longest), dealt forwards and backwards in turn.
//
// Warps 0-15: softmax (warpgroup w: query columns 32 w ... of the block) and dK / dV output; 16-19: dQ; 20: loads;
// 21: MMA; 22: LSE and delta (in the softmax warps their latency, 1300 cycles, was part of every block).  Barriers (one phase per block i unless noted; a phase is never entered twice because every arrival for
// block i+1 follows a wait that needs block i's phase):
//   q_full/q_empty[2], do_full/do_empty   loads of Q and dO
//   k_full, k_empty, v_full, v_empty      one phase per work item
//   s_full, dp_full    MMA -> softmax     S^T, dP^T in tensor memory
//   p_full             softmax -> MMA     P^T is in tensor memory
//   ds_full, ds_empty  softmax <-> MMA    dS^T is in shared memory (and dP^T in registers) / has been read
//   dq_full, dq_empty  MMA <-> dQ warps   dQ is complete / is in registers
//   fin_full           MMA -> softmax     one phase per work item: dV, dK are complete
//   vec_full/vec_empty[2]                 LSE and delta of the block's queries
#pragma once

namespace wide {

constexpr int BB = 128;                   // rows of a key block and of a query block
constexpr int kThreads = 768;
constexpr int kTile = 2 * BB * 128;       // 128 rows of up to two 64-wide bf16 chunks
constexpr int kDqChunk = BB * 128;        // [128 q][32 fp32]
constexpr int oK = 0, oV = kTile, oQ = 2 * kTile, oDO = 4 * kTile, oDS = 5 * kTile, oDQ = 6 * kTile;
constexpr int oVec = oDQ + 2 * kDqChunk;  // -LSE*log2(e) and -delta of two query blocks
constexpr int oBar = oVec + 2 * 2 * BB * 4;
constexpr int kNumBars = 4 + 4 + 2 + 2 + 1 + 2 + 2 + 1 + 4;
constexpr int kSmem = oBar + kNumBars * 8 + 16;
static_assert(kSmem <= 232448, "attention backward: shared memory over the per-CTA limit");

struct Sched {
  int nblk;         // key blocks
  int units;        // head units (dK / dV heads) per sample
  int unit_heads;   // query heads of a unit
  int bu;           // batch * units
  int group;        // head units that are walked together
  int total;
};

struct Work {
  int batch, unit, kv0, sq_b, sk_b, coff, i_start, per_head, n_iter;
};

__device__ __forceinline__ int work_index(int n) {
  return n * gridDim.x + ((n & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}

__device__ __forceinline__ Work work_at(const BwdParams& p, const Sched& s, int t) {
  Work w;
  const int per_group = s.group * s.nblk;
  const int g = t / per_group, r = t - g * per_group;
  const int gsize = min(s.group, s.bu - g * s.group);
  const int jb = r / gsize;
  const int bu = g * s.group + (r - jb * gsize);
  w.batch = bu / s.units;
  w.unit = bu - w.batch * s.units;
  // real tokens of this sample (right-padded batches); the tensors keep their padded extents p.sq / p.sk
  w.sq_b = p.seqlens_q ? min(p.sq, p.seqlens_q[w.batch]) : p.sq;
  w.sk_b = p.seqlens_k ? min(p.sk, p.seqlens_k[w.batch]) : p.sk;
  w.kv0 = jb * BB;
  w.coff = w.sk_b - w.sq_b;
  w.i_start = 0;
  if (p.causal) {
    const int first_q = w.kv0 - w.coff;      // first query row that sees key kv0
    w.i_start = first_q <= 0 ? 0 : first_q / BB;
  }
  w.per_head = w.kv0 < w.sk_b ? max(0, (w.sq_b + BB - 1) / BB - w.i_start) : 0;
  w.n_iter = w.per_head * s.unit_heads;
  return w;
}

__device__ __forceinline__ void store16(__nv_bfloat16* dst, const uint32_t* v, float scale, bool wide_store) {
  float f[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]) * scale;
  const mb::bf16x8 a = mb::pack8(f), b = mb::pack8(f + 8);
  if (wide_store) {
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

template <bool kAlias>
__global__ void __launch_bounds__(kThreads, 1)
attn_bwd_wide_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_dq, const BwdParams p, const Sched sch) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + oBar);
  uint64_t* k_full = bars;
  uint64_t* k_empty = bars + 1;
  uint64_t* v_full = bars + 2;
  uint64_t* v_empty = bars + 3;
  uint64_t* q_full = bars + 4;
  uint64_t* q_empty = bars + 6;
  uint64_t* do_full = bars + 8;
  uint64_t* do_empty = bars + 9;
  uint64_t* s_full = bars + 10;
  uint64_t* dp_full = bars + 11;
  uint64_t* p_full = bars + 12;
  uint64_t* ds_full = bars + 13;
  uint64_t* ds_empty = bars + 14;
  uint64_t* dq_full = bars + 15;
  uint64_t* dq_empty = bars + 16;
  uint64_t* fin_full = bars + 17;
  uint64_t* vec_full = bars + 18;
  uint64_t* vec_empty = bars + 20;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kNumBars);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) report(p.status, MB_ERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < kNumBars; ++i) {
      const uint64_t* b = bars + i;
      mbar_init(bars + i, (b == p_full || b == ds_full || b >= vec_empty) ? 16 : (b == dq_empty ? 4 : 1));   // warps
    }
    fence_barrier_init();
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    prefetch_tmap(&tm_do);
    prefetch_tmap(&tm_dq);
  }
  if (warp == 20) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t t_s = tmem_base, t_dp = tmem_base + 128;
  const uint32_t t_dq = kAlias ? t_dp : tmem_base + 256;
  const uint32_t t_dv = tmem_base + (kAlias ? 256 : 336), t_dk = tmem_base + (kAlias ? 384 : 416);
  constexpr uint32_t kChunk = BB * 128;

  // Registers: 768 threads were launched with 80 each; 512 * 64 + 128 * 160 + 128 * 64 is the same sum.
  if (warp >= 20) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;\n");
    if (warp == 20) {
      // --------------------------------------------------------- TMA producer
      if (lane == 0) {
        int n = 0, items = 0;                // query blocks and work items so far
        bool ok = true;
        auto load = [&](int off, const CUtensorMap* tm, uint64_t* full, uint64_t* empty, int uses, int head, int row,
                        int batch) {
          if (!ok) return;
          if (uses > 0 && !mbar_wait(empty, (uses - 1) & 1)) {
            report(p.status, MB_ERR_TIMEOUT_EMPTY);
            ok = false;
            return;
          }
          mbar_expect_tx(full, p.nchunks * kChunk);
          for (int c = 0; c < p.nchunks; ++c) tma_load_4d(smem + off + c * kChunk, tm, full, 64 * c, head, row, batch);
        };
        for (int r = 0; ok; ++r) {
          const int t = work_index(r);
          if (t >= sch.total) break;
          const Work w = work_at(p, sch, t);
          if (w.n_iter == 0) continue;
          const int head0 = w.unit * sch.unit_heads, head_kv = head0 / (p.nh / p.nh_kv);
          load(oK, &tm_k, k_full, k_empty, items, head_kv, w.kv0, w.batch);
          int hh = 0, i = 0;
          for (int it = 0; it < w.n_iter && ok; ++it) {
            const int st = n & 1, q0 = (w.i_start + i) * BB;
            load(oQ + st * kTile, &tm_q, &q_full[st], &q_empty[st], n >> 1, head0 + hh, q0, w.batch);
            if (it == 0) load(oV, &tm_v, v_full, v_empty, items, head_kv, w.kv0, w.batch);
            load(oDO, &tm_do, do_full, do_empty, n, head0 + hh, q0, w.batch);
            ++n;
            if (++i == w.per_head) { i = 0; ++hh; }
          }
          ++items;
        }
      }
    } else if (warp == 22) {
      // ------------------------------------------- LSE and delta of every query block
      float* s_vec = reinterpret_cast<float*>(smem + oVec);
      int n = 0;
      bool ok = true;
      for (int r = 0; ok; ++r) {
        const int t = work_index(r);
        if (t >= sch.total) break;
        const Work w = work_at(p, sch, t);
        int hh = 0, i = 0;
        for (int it = 0; it < w.n_iter; ++it, ++n) {
          const long row = (static_cast<long>(w.batch) * p.nh + w.unit * sch.unit_heads + hh) * p.sq;
          const int q = (w.i_start + i) * BB + lane;
          float lse[4], delta[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in = q + 32 * u < w.sq_b;
            lse[u] = in ? p.lse[row + q + 32 * u] : 0.f;
            delta[u] = in ? p.delta[row + q + 32 * u] : 0.f;
          }
          if (n >= 2 && !mbar_wait(&vec_empty[n & 1], ((n >> 1) - 1) & 1)) {
            report(p.status, MB_ERR_TIMEOUT_EMPTY);
            ok = false;
            break;
          }
          float* dst = s_vec + (n & 1) * 2 * BB + lane;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            dst[32 * u] = lse[u] * -1.4426950408889634f;
            dst[BB + 32 * u] = -delta[u];
          }
          mbar_arrive_warp(&vec_full[n & 1]);
          if (++i == w.per_head) { i = 0; ++hh; }
        }
      }
    } else if (warp == 21) {
      // ----------------------------------------------------------- MMA issuer
      const uint32_t idesc_s = make_idesc_bf16(128, BB, 0, 0);         // S^T, dP^T
      const uint32_t idesc_dkv = make_idesc_bf16(128, p.d, 0, 1);      // dV, dK
      const uint32_t idesc_dq = make_idesc_bf16(128, p.d, 1, 1);       // dQ
      const uint32_t base = smem_u32(smem);
      const int ksteps = p.d / 16;
      int n = 0, items = 0;
      bool ok = true;
      auto wait = [&](uint64_t* bar, int phase, int code) -> bool {
        if (ok && !mbar_wait(bar, phase & 1)) {
          report(p.status, code);
          ok = false;
        }
        return ok;
      };
      // both operands K-major over the head size
      auto product_kk = [&](uint32_t d_tmem, uint32_t a, uint32_t b) {
        const uint64_t da = make_smem_desc_sw128(a, 16, 1024), db = make_smem_desc_sw128(b, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = ((kk >> 2) * kChunk + (kk & 3) * 32) >> 4;
          if (kk < ksteps) mma_f16_ss(d_tmem, da + off, db + off, idesc_s, kk != 0 ? 1u : 0u);
        }
      };
      auto issue_s = [&](int nn) {
        if (!wait(&q_full[nn & 1], nn >> 1, MB_ERR_TIMEOUT_FULL)) return;
        tc_fence_after();
        if (elect_one()) {
          product_kk(t_s, base + oK, base + oQ + (nn & 1) * kTile);
          mma_commit(s_full);
        }
        __syncwarp();
      };
      auto issue_dp = [&](int nn, bool last) {
        if (!wait(do_full, nn, MB_ERR_TIMEOUT_FULL)) return;
        // dP^T of the block before is in registers (its ds_full was waited for); where dQ of that block took
        // these columns, it has to be read too
        if (kAlias && nn > 0 && !wait(dq_empty, nn - 1, MB_ERR_TIMEOUT_TMEM)) return;
        tc_fence_after();
        if (elect_one()) {
          product_kk(t_dp, base + oV, base + oDO);
          mma_commit(dp_full);
          if (last) mma_commit(v_empty);
        }
        __syncwarp();
      };
      for (int r = 0; ok; ++r) {
        const int t = work_index(r);
        if (t >= sch.total) break;
        const Work w = work_at(p, sch, t);
        if (w.n_iter == 0) continue;
        if (!wait(k_full, items, MB_ERR_TIMEOUT_FULL)) break;
        issue_s(n);
        if (!wait(v_full, items, MB_ERR_TIMEOUT_FULL)) break;
        issue_dp(n, w.n_iter == 1);
        for (int it = 0; it < w.n_iter && ok; ++it, ++n) {
          const bool next = it + 1 < w.n_iter;
          if (!wait(p_full, n, MB_ERR_TIMEOUT_TMEM)) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t d_do = make_smem_desc_sw128(base + oDO, kChunk, 1024);
#pragma unroll
            for (int kk = 0; kk < BB / 16; ++kk)
              // P^T of query columns 32 w ... lies over the first half of those S^T columns
              mma_f16_ts(t_dv, t_s + (kk >> 1) * 32 + (kk & 1) * 8, d_do + kk * (2048 >> 4), idesc_dkv, (it | kk) != 0);
            mma_commit(do_empty);
          }
          __syncwarp();
          if (next) issue_s(n + 1);
          if (!wait(ds_full, n, MB_ERR_TIMEOUT_TMEM)) break;
          tc_fence_after();
          auto issue_dk = [&]() {
            const uint64_t d_ds_k = make_smem_desc_sw128(base + oDS, 16, 1024);
            const uint64_t d_q_mn = make_smem_desc_sw128(base + oQ + (n & 1) * kTile, kChunk, 1024);
#pragma unroll
            for (int kk = 0; kk < BB / 16; ++kk)
              mma_f16_ss(t_dk, d_ds_k + (((kk >> 2) * kChunk + (kk & 3) * 32) >> 4), d_q_mn + kk * (2048 >> 4), idesc_dkv,
                         (it | kk) != 0);
            mma_commit(&q_empty[n & 1]);
          };
          auto issue_dq = [&]() {
            const uint64_t d_ds_mn = make_smem_desc_sw128(base + oDS, kChunk, 1024);
            const uint64_t d_k_mn = make_smem_desc_sw128(base + oK, kChunk, 1024);
#pragma unroll
            for (int kk = 0; kk < BB / 16; ++kk)
              mma_f16_ss(t_dq, d_ds_mn + kk * (2048 >> 4), d_k_mn + kk * (2048 >> 4), idesc_dq, kk != 0);
            mma_commit(dq_full);
            if (!next) mma_commit(k_empty);
          };
          if (kAlias) {          // dQ first: dP^T of the next block waits for its columns
            if (elect_one()) {
              issue_dq();
              issue_dk();
              mma_commit(ds_empty);
              if (!next) mma_commit(fin_full);
            }
            __syncwarp();
            if (next) issue_dp(n + 1, it + 2 == w.n_iter);
          } else {               // dP^T of the next block, which the softmax warps wait for, as soon as its dO can be there
            if (elect_one()) issue_dk();
            __syncwarp();
            if (next) issue_dp(n + 1, it + 2 == w.n_iter);
            if (n > 0 && !wait(dq_empty, n - 1, MB_ERR_TIMEOUT_TMEM)) break;
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
              issue_dq();
              mma_commit(ds_empty);
              if (!next) mma_commit(fin_full);
            }
            __syncwarp();
          }
        }
        ++items;
      }
    }
  } else if (warp >= 16) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;\n");
    // ------------------------------------- dQ: tensor memory -> staging -> TMA reduce-add
    const int r = threadIdx.x & 127;               // query row == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool leader = (r == 0);
    uint8_t* sdq_ = smem + oDQ;
    const int nw = (p.d + 31) / 32;
    int n = 0, buf = 0;
    bool ok = true;
    for (int rnd = 0; ok; ++rnd) {
      const int t = work_index(rnd);
      if (t >= sch.total) break;
      const Work w = work_at(p, sch, t);
      int hh = 0, i = 0;
      for (int it = 0; it < w.n_iter; ++it, ++n) {
        if (!mbar_wait(dq_full, n & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t qr[128];
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (c < nw) tmem_ld32(t_dq + 32 * c + lane_off, qr + 32 * c);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive_warp(dq_empty);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c >= nw) break;
          if (leader) tma_wait_read<1>();          // the reduce before last has read this staging chunk
          asm volatile("bar.sync 2, 128;" ::: "memory");
          uint8_t* row = sdq_ + buf * kDqChunk + r * 128;
#pragma unroll
          for (int g = 0; g < 8; ++g)
            *reinterpret_cast<uint4*>(row + ((g ^ (r & 7)) << 4)) =
                make_uint4(qr[32 * c + 4 * g], qr[32 * c + 4 * g + 1], qr[32 * c + 4 * g + 2], qr[32 * c + 4 * g + 3]);
          fence_async_smem();
          asm volatile("bar.sync 2, 128;" ::: "memory");
          if (leader) {
            asm volatile(
                "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group "
                "[%0, {%2, %3, %4}], [%1];\n" ::"l"(reinterpret_cast<uint64_t>(&tm_dq)),
                "r"(smem_u32(sdq_ + buf * kDqChunk)), "r"(32 * c), "r"((w.i_start + i) * BB),
                "r"(w.batch * p.nh + w.unit * sch.unit_heads + hh)
                : "memory");
            tma_commit();
          }
          buf ^= 1;
        }
        if (++i == w.per_head) { i = 0; ++hh; }
      }
    }
    if (leader) tma_wait_all<0>();
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;\n");
    // ------------------------------------------------------ softmax / dS / dK, dV output
    const int r = threadIdx.x & 127;               // key row == TMEM lane
    const int part = threadIdx.x >> 7;             // query columns 32 * part ...
    const int c0 = part * 32;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    uint8_t* sds_ = smem + oDS + (part >> 1) * kChunk + r * 128;
    float* s_vec = reinterpret_cast<float*>(smem + oVec);      // [buffer][lse, delta][128]
    const mb::f32x2 scale2 = mb::pack_f32x2(p.scale_log2, p.scale_log2);
    const bool wide_store =
        (((reinterpret_cast<uintptr_t>(p.dk) | reinterpret_cast<uintptr_t>(p.dv)) & 31) |
         ((p.dk_bs | p.dk_ts | p.dk_hs | p.dv_bs | p.dv_ts | p.dv_hs) & 15)) == 0;
    int n = 0, items = 0;
    bool ok = true;
    for (int rnd = 0; ok; ++rnd) {
      const int t = work_index(rnd);
      if (t >= sch.total) break;
      const Work w = work_at(p, sch, t);
      const int kv_idx = w.kv0 + r, kv_last = w.kv0 + BB - 1;
      int i = 0;
      for (int it = 0; it < w.n_iter; ++it, ++n) {
        const int q0 = (w.i_start + i) * BB;
        if (++i == w.per_head) i = 0;
        const float* v_lse = s_vec + (n & 1) * 2 * BB + c0;
        const float* v_delta = v_lse + BB;
        if (!mbar_wait(&vec_full[n & 1], (n >> 1) & 1) || !mbar_wait(s_full, n & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        tc_fence_after();
        uint32_t pf[32];                           // S^T, then P^T in fp32
        tmem_ld32(t_s + c0 + lane_off, pf);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          const ulonglong2 l2 = *reinterpret_cast<const ulonglong2*>(v_lse + c);
          const float2 xa = mb::unpack_f32x2(
              mb::fma_f32x2(mb::pack_f32x2(__uint_as_float(pf[c]), __uint_as_float(pf[c + 1])), scale2, l2.x));
          const float2 xb = mb::unpack_f32x2(
              mb::fma_f32x2(mb::pack_f32x2(__uint_as_float(pf[c + 2]), __uint_as_float(pf[c + 3])), scale2, l2.y));
          pf[c] = __float_as_uint(mb::fast_exp2(xa.x));
          pf[c + 1] = __float_as_uint(mb::fast_exp2(xa.y));
          pf[c + 2] = __float_as_uint(mb::fast_exp2(xb.x));
          pf[c + 3] = __float_as_uint(mb::fast_exp2(xb.y));
        }
        if ((q0 + BB > w.sq_b) || (kv_last >= w.sk_b) || (p.causal && kv_last > q0 + w.coff)) {
          // visible columns of this key row: lo <= c < hi
          const int lo = p.causal ? kv_idx - w.coff - q0 - c0 : 0;
          const int hi = kv_idx < w.sk_b ? w.sq_b - q0 - c0 : 0;
#pragma unroll
          for (int c = 0; c < 32; ++c) pf[c] = (c >= lo && c < hi) ? pf[c] : 0u;
        }
        {
          uint32_t pk[16];
#pragma unroll
          for (int c = 0; c < 32; c += 2) pk[c >> 1] = pack2(__uint_as_float(pf[c]), __uint_as_float(pf[c + 1]));
          tmem_st16(t_s + c0 + lane_off, pk);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(p_full);

        if (!mbar_wait(dp_full, n & 1) || (n > 0 && !mbar_wait(ds_empty, (n - 1) & 1))) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t dr[16], ds[8];
          tmem_ld16(t_dp + c0 + 16 * h + lane_off, dr);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; c += 4) {
            const ulonglong2 d2 = *reinterpret_cast<const ulonglong2*>(v_delta + 16 * h + c);
            const uint32_t* pp = pf + 16 * h + c;
            const float2 a = mb::unpack_f32x2(mb::mul_f32x2(
                mb::pack_f32x2(__uint_as_float(pp[0]), __uint_as_float(pp[1])),
                mb::add_f32x2(mb::pack_f32x2(__uint_as_float(dr[c]), __uint_as_float(dr[c + 1])), d2.x)));
            const float2 b = mb::unpack_f32x2(mb::mul_f32x2(
                mb::pack_f32x2(__uint_as_float(pp[2]), __uint_as_float(pp[3])),
                mb::add_f32x2(mb::pack_f32x2(__uint_as_float(dr[c + 2]), __uint_as_float(dr[c + 3])), d2.y)));
            ds[c >> 1] = pack2(a.x, a.y);
            ds[(c >> 1) + 1] = pack2(b.x, b.y);
          }
#pragma unroll
          for (int g = 0; g < 2; ++g)
            *reinterpret_cast<uint4*>(sds_ + (((4 * (part & 1) + 2 * h + g) ^ (r & 7)) << 4)) =
                make_uint4(ds[4 * g], ds[4 * g + 1], ds[4 * g + 2], ds[4 * g + 3]);
        }
        fence_async_smem();
        tc_fence_before();
        mbar_arrive_warp(ds_full);
        mbar_arrive_warp(&vec_empty[n & 1]);
      }
      if (!ok) break;

      if (w.n_iter > 0) {
        if (!mbar_wait(fin_full, items & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        ++items;
        tc_fence_after();
      }
      __nv_bfloat16* dkrow = p.dk + w.batch * p.dk_bs + static_cast<long>(kv_idx) * p.dk_ts + w.unit * p.dk_hs;
      __nv_bfloat16* dvrow = p.dv + w.batch * p.dv_bs + static_cast<long>(kv_idx) * p.dv_ts + w.unit * p.dv_hs;
      for (int c = part * 16; c < p.d; c += 64) {
        uint32_t a[16], b[16];
        if (w.n_iter > 0) {
          tmem_ld16(t_dv + c + lane_off, a);
          tmem_ld16(t_dk + c + lane_off, b);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int u = 0; u < 16; ++u) a[u] = b[u] = 0;
        }
        if (kv_idx < p.sk) {
          store16(dvrow + c, a, 1.f, wide_store);
          store16(dkrow + c, b, p.scale, wide_store);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 20) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace wide
