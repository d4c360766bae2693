// Attention forward for short sequences; included by attn_fwd_tcgen05.cu.
//
// One CTA owns a 128-row query tile of one (batch, head) and walks the keys in blocks of 64; both products of a block
// run on tcgen05.mma with their accumulators in tensor memory:
//   S  = Q K^T   (A = Q K-major, B = K K-major)                        two buffers
//   O += P V     (A = P K-major from shared memory, B = V MN-major)
// Warps 0-3 do the softmax (one query row per thread), warp 4 issues the loads, warp 5 the MMAs.  Two CTAs fit an SM.
//
// What bounds a sequence of a block or two is the chain from its loads to its output, 3 - 4 us: many of them have to be
// under way at once, and a second query tile per CTA would stand empty.  The persistent kernel keeps one work item per SM
// in flight: 256 x 8 heads of 32, 16 queries and 64 keys 48.1 us, this one 28.9; 64 x 16 heads of 64, 32 x 32 positions
// 27.2 us and 17.9.
#pragma once

namespace one_tile {

constexpr int BN = 64;
constexpr int kThreads = 192;
constexpr int kStages = 2;

struct Smem {
  // every tile is a stack of [rows][64 bf16] chunks, 128-byte swizzled
  static constexpr int kQ = 2 * BM * 128;           // up to 2 chunks
  static constexpr int kKV = 2 * BN * 128;          // one stage of K or V
  static constexpr int kP = (BN / 64) * BM * 128;
  static constexpr int oQ = 0;
  static constexpr int oK = oQ + kQ;
  static constexpr int oV = oK + kStages * kKV;
  static constexpr int oP = oV + kStages * kKV;
  static constexpr int oBar = oP + kP;
  // q_full, k_full[2], v_full[2], kv_empty[2], s_full[2], s_empty[2], p_full, pv_done, k_empty[2]
  static constexpr int kNumBars = 1 + 2 + 2 + 2 + 2 + 2 + 1 + 1 + 2;
  static constexpr int kTotal = oBar + kNumBars * 8 + 16;
};

__global__ void __launch_bounds__(kThreads, 2)
attn_fwd_one_tile_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                         const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
  using L = Smem;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::oBar);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* v_full = bars + 3;
  uint64_t* kv_empty = bars + 5;
  uint64_t* s_full = bars + 7;
  uint64_t* s_empty = bars + 9;
  uint64_t* p_full = bars + 11;
  uint64_t* pv_done = bars + 12;
  uint64_t* k_empty = bars + 13;   // K stage free as soon as its S MMA has read it (V waits for PV)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::kNumBars);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // heavy (late) query tiles first: under the causal mask they have the most blocks
  const int qt = gridDim.x - 1 - blockIdx.x;
  const int head = blockIdx.y;
  const int batch = blockIdx.z;
  const int head_kv = head / (p.nh / p.nh_kv);
  const int q0 = qt * BM;
  const int sq_b = p.seqlens_q ? min(p.sq, p.seqlens_q[batch]) : p.sq;   // real tokens of this sample
  const int sk_b = p.seqlens_k ? min(p.sk, p.seqlens_k[batch]) : p.sk;
  const int coff = sk_b - sq_b;  // causal: key j visible to query i when j <= i + coff

  int nblocks = (q0 < sq_b) ? (sk_b + BN - 1) / BN : 0;   // a tile of padding rows has nothing to attend to
  if (p.causal) {
    int last = q0 + BM - 1 + coff;  // last visible key of the tile's last row
    int nb = last < 0 ? 0 : last / BN + 1;
    nblocks = min(nblocks, nb);
  }

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled tiles need a 1024-byte base
    if (threadIdx.x == 0) report(p.status, MB_ERR_BAD_ARG);
    return;
  }

  constexpr int kTmemCols = 256;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&kv_empty[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], 128);
    }
    mbar_init(p_full, 128);
    mbar_init(pv_done, 1);
    fence_barrier_init();
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
  }
  if (warp == 4) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_s = tmem_base;           // S0 at +0, S1 at +BN
  const uint32_t tmem_o = tmem_base + 2 * BN;  // O accumulator

  const uint32_t chunk_q = BM * 128, chunk_kv = BN * 128;

  if (warp == 4) {
    // ----------------------------------------------------------- TMA producer
    if (lane == 0 && nblocks > 0) {
      bool ok = true;
      mbar_expect_tx(q_full, p.nchunks * chunk_q);
      for (int c = 0; c < p.nchunks; ++c)
        tma_load_4d(smem + L::oQ + c * chunk_q, &tm_q, q_full, 64 * c, head, q0, batch);
      for (int j = 0; j < nblocks && ok; ++j) {
        int st = j % kStages;
        if (j >= kStages && !mbar_wait(&k_empty[st], ((j / kStages) - 1) & 1)) {
          report(p.status, MB_ERR_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        uint8_t* sk_ = smem + L::oK + st * L::kKV;
        uint8_t* sv_ = smem + L::oV + st * L::kKV;
        mbar_expect_tx(&k_full[st], p.nchunks * chunk_kv);
        for (int c = 0; c < p.nchunks; ++c)
          tma_load_4d(sk_ + c * chunk_kv, &tm_k, &k_full[st], 64 * c, head_kv, j * BN, batch);
        if (j >= kStages && !mbar_wait(&kv_empty[st], ((j / kStages) - 1) & 1)) {
          report(p.status, MB_ERR_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        mbar_expect_tx(&v_full[st], p.nchunks * chunk_kv);
        for (int c = 0; c < p.nchunks; ++c)
          tma_load_4d(sv_ + c * chunk_kv, &tm_v, &v_full[st], 64 * c, head_kv, j * BN, batch);
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------- MMA issuer
    if (nblocks > 0) {
      const uint32_t idesc_s = make_idesc_bf16(BM, BN, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(BM, p.d_mma, 0, 1);
      const uint32_t sq_ = smem_u32(smem + L::oQ);
      const uint32_t sp_ = smem_u32(smem + L::oP);
      const int ksteps = p.d_mma / 16;
      bool ok = true;

      auto issue_s = [&](int j) -> bool {
        int st = j % kStages, b = j & 1;
        if (!mbar_wait(&k_full[st], (j / kStages) & 1)) return false;
        if (j >= 2 && !mbar_wait(&s_empty[b], ((j >> 1) - 1) & 1)) return false;
        tc_fence_after();
        if (elect_one()) {
          uint32_t sk_ = smem_u32(smem + L::oK + st * L::kKV);
          for (int kk = 0; kk < ksteps; ++kk) {
            uint32_t ch = kk >> 2, in = (kk & 3) * 32;
            uint64_t ad = make_smem_desc_sw128(sq_ + ch * chunk_q + in, 16, 1024);
            uint64_t bd = make_smem_desc_sw128(sk_ + ch * chunk_kv + in, 16, 1024);
            mma_f16_ss(tmem_s + b * BN, ad, bd, idesc_s, kk != 0 ? 1u : 0u);
          }
          mma_commit(&k_empty[st]);
          mma_commit(&s_full[b]);
        }
        __syncwarp();
        return true;
      };

      if (!mbar_wait(q_full, 0)) { report(p.status, MB_ERR_TIMEOUT_FULL); ok = false; }
      if (ok && !issue_s(0)) { report(p.status, MB_ERR_TIMEOUT_FULL); ok = false; }
      for (int j = 0; j < nblocks && ok; ++j) {
        if (j + 1 < nblocks && !issue_s(j + 1)) {
          report(p.status, MB_ERR_TIMEOUT_FULL);
          ok = false;
          break;
        }
        int st = j % kStages;
        if (!mbar_wait(p_full, j & 1) || !mbar_wait(&v_full[st], (j / kStages) & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
          uint32_t sv_ = smem_u32(smem + L::oV + st * L::kKV);
#pragma unroll
          for (int kk = 0; kk < BN / 16; ++kk) {
            uint32_t ch = kk >> 2, in = (kk & 3) * 32;
            uint64_t ad = make_smem_desc_sw128(sp_ + ch * chunk_q + in, 16, 1024);
            // V: [kv rows][64-wide d atoms]; 16 kv rows = 2048 B, next d atom = chunk_kv
            uint64_t bd = make_smem_desc_sw128(sv_ + kk * 2048, chunk_kv, 1024);
            mma_f16_ss(tmem_o, ad, bd, idesc_o, (j | kk) != 0 ? 1u : 0u);
          }
          mma_commit(&kv_empty[st]);
          mma_commit(pv_done);
        }
        __syncwarp();
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax
    const int r = threadIdx.x;  // row of the tile == TMEM lane
    const int qi = q0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(warp * 32) << 16;
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    uint8_t* sp_ = smem + L::oP;

    for (int j = 0; j < nblocks && ok; ++j) {
      const int b = j & 1;
      if (!mbar_wait(&s_full[b], (j >> 1) & 1)) {
        report(p.status, MB_ERR_TIMEOUT_TMEM);
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sr[BN];
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) tmem_ld32(tmem_s + b * BN + c * 32 + lane_off, sr + 32 * c);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(&s_empty[b]);

      const int kv0 = j * BN;
      const int vis = p.causal ? min(sk_b - 1, qi + coff) : sk_b - 1;  // last visible key
      // Only tiles that touch the diagonal or the end of the keys need the mask; the test is the
      // same for every thread of the CTA (first row of the tile has the smallest horizon).
      const int vis_tile = p.causal ? min(sk_b - 1, q0 + coff) : sk_b - 1;
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
      if (kv0 + BN - 1 > vis_tile) {
#pragma unroll
        for (int i = 0; i < BN; i += 4) {
          float v0 = (kv0 + i <= vis) ? __uint_as_float(sr[i]) : -INFINITY;
          float v1 = (kv0 + i + 1 <= vis) ? __uint_as_float(sr[i + 1]) : -INFINITY;
          float v2 = (kv0 + i + 2 <= vis) ? __uint_as_float(sr[i + 2]) : -INFINITY;
          float v3 = (kv0 + i + 3 <= vis) ? __uint_as_float(sr[i + 3]) : -INFINITY;
          sr[i] = __float_as_uint(v0); sr[i + 1] = __float_as_uint(v1);
          sr[i + 2] = __float_as_uint(v2); sr[i + 3] = __float_as_uint(v3);
          mx0 = fmaxf(mx0, v0); mx1 = fmaxf(mx1, v1); mx2 = fmaxf(mx2, v2); mx3 = fmaxf(mx3, v3);
        }
      } else {
#pragma unroll
        for (int i = 0; i < BN; i += 4) {
          mx0 = fmaxf(mx0, __uint_as_float(sr[i]));
          mx1 = fmaxf(mx1, __uint_as_float(sr[i + 1]));
          mx2 = fmaxf(mx2, __uint_as_float(sr[i + 2]));
          mx3 = fmaxf(mx3, __uint_as_float(sr[i + 3]));
        }
      }
      // raw scores; the softmax scale (> 0, so maxima commute with it) is folded into the FFMA below
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * p.scale_log2;
      // Lazy rescaling: keep the old reference maximum unless the new one is much
      // larger; probabilities then stay below 2^8, harmless in fp32 / bf16.
      const float m_new = fmaxf(m_run, mx);
      const float m_use = (m_new - m_run > 8.f || m_run == -INFINITY) ? m_new : m_run;
      const float alpha = (m_run == -INFINITY) ? 0.f : exp2f(m_run - m_use);
      const float m_neg = (m_use == -INFINITY) ? 0.f : -m_use;
      float sum0 = 0.f, sum1 = 0.f;
      uint32_t pk[BN / 2];
#pragma unroll
      for (int i = 0; i < BN; i += 2) {
        const float xa = fmaf(__uint_as_float(sr[i]), p.scale_log2, m_neg);
        const float xc = fmaf(__uint_as_float(sr[i + 1]), p.scale_log2, m_neg);
        const float a = mb::fast_exp2(xa);
        const float c = mb::fast_exp2(xc);
        sum0 += a;
        sum1 += c;
        pk[i >> 1] = pack_bf16x2(a, c);
      }
      const float sum = sum0 + sum1;
      l_run = l_run * alpha + sum;
      m_run = m_use;

      if (j > 0) {
        if (!mbar_wait(pv_done, (j - 1) & 1)) {
          report(p.status, MB_ERR_TIMEOUT_TMEM);
          ok = false;
          break;
        }
        tc_fence_after();
      }
      // P tile -> shared memory in the swizzled K-major layout the MMA reads
#pragma unroll
      for (int g = 0; g < BN / 8; ++g) {
        uint32_t ch = g >> 3, gg = g & 7;
        uint4 val = make_uint4(pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]);
        *reinterpret_cast<uint4*>(sp_ + ch * chunk_q + r * 128 + ((gg ^ (r & 7)) << 4)) = val;
      }
      // Rescale the running output when this warp's reference maxima moved.
      const bool need = (j > 0) && (alpha != 1.f);
      if (__any_sync(0xffffffffu, need)) {
        for (int c = 0; c < p.d_mma / 16; ++c) {
          uint32_t o[16];
          tmem_ld16(tmem_o + c * 16 + lane_off, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st16(tmem_o + c * 16 + lane_off, o);
        }
        tmem_st_wait();
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(p_full);
    }

    if (ok && nblocks > 0) {
      if (!mbar_wait(pv_done, (nblocks - 1) & 1)) {
        report(p.status, MB_ERR_TIMEOUT_TMEM);
        ok = false;
      }
    }
    if (ok) {
      tc_fence_after();
      const bool real_row = qi < sq_b;
      const float inv = (real_row && l_run > 0.f) ? 1.f / l_run : 0.f;
      __nv_bfloat16* orow = p.o + batch * p.o_batch_stride + static_cast<long>(qi) * p.o_tok_stride +
                            static_cast<long>(head) * p.o_head_stride;
      for (int c = 0; c < p.d_mma / 16; ++c) {
        uint32_t o[16];
        if (nblocks > 0) {
          tmem_ld16(tmem_o + c * 16 + lane_off, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = 0;
        }
        if (qi < p.sq && c * 16 < p.d) {
          float f[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(o[i]) * inv;
          *reinterpret_cast<mb::bf16x8*>(orow + c * 16) = mb::pack8(f);
          *reinterpret_cast<mb::bf16x8*>(orow + c * 16 + 8) = mb::pack8(f + 8);
        }
      }
      if (qi < p.sq)
        p.lse[(static_cast<long>(batch) * p.nh + head) * p.sq + qi] =
            (real_row && l_run > 0.f) ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Where this kernel beats the persistent one; both measured for 1 - 512 queries, 16 - 1024 keys, 8 - 4096 (batch, head)s
// and head sizes 32 - 128 (646 cases).  Outside of the rule the persistent kernel is at most 8 % slower, and up to three
// times as fast.
bool is_faster(int sq, int sk, long heads, int d) {
  const long tiles = (sq + BM - 1) / BM * heads;
  if (sq <= 32 && sk <= 256) return true;
  if (sq <= 64 && sk <= 64 && (d <= 64 || (heads > 148 && heads <= 600))) return true;
  if (heads > 148) {           // the persistent kernel needs a second round
    if (sq <= 32) return sk <= 1024;
    if (sq <= 64 && heads <= 296) return sk <= 512;
    if (d <= 64 && sq <= (d <= 32 ? 128 : 64)) return sk <= 512;
  }
  // tiles that all run at once, each on an SM of its own
  return d <= 64 && sq > BM && sk <= (d <= 32 ? 320 : 192) && tiles <= 148;
}

}  // namespace one_tile
