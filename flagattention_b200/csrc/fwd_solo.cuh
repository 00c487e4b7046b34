// Forward attention for head dimensions up to 64: one 128-row query tile per block, several blocks per SM.
//
// fwd_kernel (fwd_kernel.cuh) pairs two query tiles in one block per SM. At D = 128 the accumulators and scores fill
// TMEM that way; at D <= 64 they fill 384 of the 512 columns, the products are half as long and the eight softmax warps
// of an SM are what its time goes to, waiting for their own latencies (0.52 instructions issued per scheduler and
// cycle). Here a block is one tile with four softmax warps and 128 columns of TMEM (64 scores and the accumulator), so
// SOLO_BLOCKS of them share an SM: their softmax chains fill each other's gaps, and start-up, first loads and output
// of a short item run under the others' work without any chaining of items.
//
// Roles: warps 0-3 softmax and epilogue (thread r <-> row r <-> TMEM lane r), warp 4 tcgen05.mma, warp 5 TMA (6 and 7
// idle). A step is
// 64 keys: S = Q K^T, P (16-bit) over the first 32 columns of S, O += P V. Issue order P V (u), Q K^T (u + 1): the
// tensor pipe executes in order, so S of step u + 1 also certifies that O of step u is complete.
//
// Numerics: P is rounded to 16 bits against the running maximum, which is lazy (RESCALE_THRESHOLD) except within a row's
// first 128 keys. There the second step takes the larger maximum over at once, so that the largest probability of a
// short row is 1 and rounds exactly, as it does in fwd_kernel, whose steps are 128 keys. (Lazy there too, the error of O
// against float64 was 0.4 to 1 % larger than fwd_kernel's at 512 to 2048 keys and 2.3 to 4.7 % at 128.)
#pragma once
#include "fwd_kernel.cuh"

namespace b200attn {

// Per SM. Three measured 2 to 5 % slower although they spill nothing (four: 32 to 52 bytes stored and 64 to 152 loaded a
// thread): the schedulers want the warps.
constexpr int SOLO_BLOCKS = 4;

template <int D>
struct SoloSmem {
  static constexpr int SUB = 64;                                // keys per step
  static constexpr int STAGES = D == 64 ? 2 : 4;
  static constexpr int SLOT_BYTES = SUB * D * 2;
  static constexpr int SLOT_CHUNK_BYTES = SUB * TileCfg<D>::ROW_BYTES;
  static constexpr int K_OFFSET = TileCfg<D>::TILE_BYTES;       // the Q tile comes first; O leaves through its place
  static constexpr int V_OFFSET = K_OFFSET + STAGES * SLOT_BYTES;
  static constexpr int BAR_OFFSET = V_OFFSET + STAGES * SLOT_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + 256 + 1024;         // barriers + alignment slack
  // Two warpgroups: the softmax group takes registers over from the other one (launched with 65536 / (256 SOLO_BLOCKS)
  // per thread; twice that is split).
  static constexpr int THREADS = 256;
  static constexpr int HELPER_REGS = 32;
  static constexpr int SOFTMAX_REGS = 2 * (65536 / (THREADS * SOLO_BLOCKS) / 8 * 8) - HELPER_REGS;
  static constexpr int TMEM_COLS = 128;
};

template <int D, bool BF16, bool DROPOUT>
__global__ void __launch_bounds__(SoloSmem<D>::THREADS, SOLO_BLOCKS)
fwd_solo_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdArgs args) {
  using Cfg = TileCfg<D>;
  using Sm = SoloSmem<D>;
  constexpr int SUB = Sm::SUB, STAGES = Sm::STAGES, BLOCK = Cfg::BLOCK;
  static_assert(SUB + D <= Sm::TMEM_COLS && Cfg::NCHUNK == 1, "head dimensions up to 64");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + Sm::K_OFFSET;
  uint8_t* sV = smem + Sm::V_OFFSET;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Sm::BAR_OFFSET);
  uint64_t* q_full = bars;                // [1]
  uint64_t* k_full = bars + 1;            // [STAGES]
  uint64_t* k_empty = k_full + STAGES;    // [STAGES]
  uint64_t* v_full = k_empty + STAGES;    // [STAGES]
  uint64_t* v_empty = v_full + STAGES;    // [STAGES]
  uint64_t* s_full = v_empty + STAGES;    // [1]
  uint64_t* p_full = s_full + 1;          // [1]
  uint64_t* o_full = p_full + 1;          // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // Work item: 128 query rows of one (batch, head), longest first; n_sub steps from key `key0` on.
  const BlockCoord bc = args.order.decode(blockIdx.x);
  const int b = args.div_heads.div(bc.bh);
  const int h = bc.bh - b * args.Hq;
  const int hk = args.div_groups.div(h);
  const int m0 = (args.n_zblocks - 1 - bc.z) * BLOCK;
  const int N = args.N, P_SEQ = args.N - args.M;
  const bool far_edge = args.causal && args.d_max < BAND_INF, near_edge = args.causal && args.d_min > -BAND_INF;
  const int key0 = far_edge ? max(0, m0 + P_SEQ - args.d_max + 1) / SUB * SUB : 0;
  const int key_hi = near_edge ? min(N, max(0, P_SEQ + m0 + BLOCK - args.d_min)) : N;
  const int n_sub = key_hi > key0 ? cdiv(key_hi - key0, SUB) : 0;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(p_full, BLOCK);
    mbar_init(o_full, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 4) {
    tmem_alloc(tmem_slot, Sm::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  pdl_wait();

  auto fail = [&](int32_t code) {
    report_status(args.status, code);
    *abort_flag = 1;
  };
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    return bounded_wait(bar, parity, abort_flag, args.status, WAIT_LIMIT_NS);
  };

  if (warp > 5) {
    reg_dealloc<Sm::HELPER_REGS>();
  } else if (warp == 5) {
    // ------------------------------------------------------------ TMA producer
    reg_dealloc<Sm::HELPER_REGS>();
    if (lane == 0 && n_sub > 0) {
      mbar_expect_tx(q_full, Cfg::TILE_BYTES);
      tma_load_4d(sQ, &tmQ, q_full, 0, m0, h, b);
      for (int u = 0; u < n_sub; ++u) {
        const int st = u % STAGES;
        const uint32_t par = ((u / STAGES) & 1) ^ 1;
        if (!wait(&k_empty[st], par)) { fail(ST_WAIT_EMPTY); break; }
        mbar_expect_tx(&k_full[st], Sm::SLOT_BYTES);
        tma_load_4d(sK + st * Sm::SLOT_BYTES, &tmK, &k_full[st], 0, key0 + u * SUB, hk, b);
        if (!wait(&v_empty[st], par)) { fail(ST_WAIT_EMPTY); break; }
        mbar_expect_tx(&v_full[st], Sm::SLOT_BYTES);
        tma_load_4d(sV + st * Sm::SLOT_BYTES, &tmV, &v_full[st], 0, key0 + u * SUB, hk, b);
      }
    }
    __syncwarp();
  } else if (warp == 4) {
    // ------------------------------------------------------------- MMA issuer (warp-uniform, see mma_ss_w)
    reg_dealloc<Sm::HELPER_REGS>();
    constexpr uint32_t IDESC_QK = make_idesc(BF16, 128, SUB, false, false);
    constexpr uint32_t IDESC_PV = make_idesc(BF16, 128, D, false, true);
    constexpr uint64_t V_DESC = make_smem_desc_hi(Sm::SLOT_CHUNK_BYTES, 8 * Cfg::ROW_BYTES, Cfg::UMMA_SWZ);
    const uint64_t dq = smem_desc(Cfg::KMAJOR_DESC, smem_u32(sQ));
    auto wait_all = [&](uint64_t* bar, uint32_t parity, int32_t code) -> bool {
      const bool w = wait(bar, parity);
      if (__all_sync(0xffffffffu, w)) return true;
      fail(code);
      return false;
    };
    auto issue_qk = [&](int st) {
      const uint64_t dk = smem_desc(Cfg::KMAJOR_DESC, smem_u32(sK) + st * Sm::SLOT_BYTES);
#pragma unroll
      for (int s = 0; s < D / 16; ++s)
        mma_ss_w(tmem_base, dq + ((s * 32) >> 4), dk + ((s * 32) >> 4), IDESC_QK, s > 0 ? 1u : 0u);
      tc_commit_w(s_full);
      tc_commit_w(&k_empty[st]);
    };
    if (n_sub > 0 && wait_all(q_full, 0, ST_WAIT_TMA) && wait_all(&k_full[0], 0, ST_WAIT_TMA)) {
      tc_fence_after();
      issue_qk(0);
      for (int u = 0; u < n_sub; ++u) {
        const int st = u % STAGES, st_next = (u + 1) % STAGES;
        const bool more = u + 1 < n_sub;
        if (!wait_all(&v_full[st], (u / STAGES) & 1, ST_WAIT_TMA)) break;
        if (more && !wait_all(&k_full[st_next], ((u + 1) / STAGES) & 1, ST_WAIT_TMA)) break;
        if (!wait_all(p_full, u & 1, ST_WAIT_SOFTMAX)) break;
        tc_fence_after();
        const uint64_t dv = smem_desc(V_DESC, smem_u32(sV) + st * Sm::SLOT_BYTES);
#pragma unroll
        for (int s = 0; s < SUB / 16; ++s)
          mma_ts_w(tmem_base + SUB, tmem_base + s * 8, dv + ((s * 16 * Cfg::ROW_BYTES) >> 4), IDESC_PV,
                   (u > 0 || s > 0) ? 1u : 0u);
        if (more) issue_qk(st_next); else tc_commit_w(o_full);
        tc_commit_w(&v_empty[st]);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------- softmax + epilogue warps
    reg_alloc<Sm::SOFTMAX_REGS>();
    const int row = warp * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_base, tmem_o = tmem_s + SUB;
    const float qk_scale = args.qk_scale;
    const int m_glob = m0 + row;
    // This row sees the keys [lo, lim); steps inside [full_from, full_upto) need no masking for any row.
    const int lim = near_edge ? min(N, max(0, P_SEQ + m_glob + 1 - args.d_min)) : N;
    const int lo = far_edge ? max(0, P_SEQ + m_glob + 1 - args.d_max) : 0;
    const int full_upto = near_edge ? min(N, max(0, P_SEQ + m0 + 1 - args.d_min)) : N;
    const int full_from = far_edge ? max(0, P_SEQ + m0 + BLOCK - args.d_max) : 0;
    uint64_t ctr_row = 0;
    const uint32_t* mk = nullptr;
    uint32_t keep_next[2] = {0u, 0u};
    if constexpr (DROPOUT) {
      const int64_t bh = static_cast<int64_t>(b) * args.Hq + h;
      ctr_row = args.drop.offset + (static_cast<uint64_t>(bh) * args.M + static_cast<uint64_t>(m_glob)) * static_cast<uint64_t>(N);
      if (args.drop.keep_mask != nullptr) mk = args.drop.keep_mask + bh * args.drop.mask_words * args.M + m_glob;
    }
    auto load_keep = [&](int n0) {
#pragma unroll
      for (int w = 0; w < 2; ++w)
        keep_next[w] = (m_glob < args.M && (n0 >> 5) + w < args.drop.mask_words)
                           ? __ldg(mk + static_cast<int64_t>((n0 >> 5) + w) * args.M) : 0u;
    };
    if constexpr (DROPOUT) {
      if (mk != nullptr && n_sub > 0) load_keep(key0);
    }
    float m_run = -INFINITY, l_run = 0.f;
    float growth = RESCALE_THRESHOLD;  // by how much this step's maximum may exceed m_run without a rescale
    bool ok = true;
    for (int u = 0; u < n_sub; ++u) {
      const int n0 = key0 + u * SUB;
      uint32_t keep_bits[DROPOUT ? 2 : 1];
      if constexpr (DROPOUT) {
        if (mk != nullptr) {
          keep_bits[0] = keep_next[0];
          keep_bits[1] = keep_next[1];
          if (u + 1 < n_sub) load_keep(n0 + SUB);
        } else {
#pragma unroll
          for (int w = 0; w < 2; ++w) keep_bits[w] = dropout_keep_word(args.drop, ctr_row + static_cast<uint64_t>(n0 + 32 * w));
        }
      }
      {
        const bool w = wait(s_full, u & 1);
        if (!__all_sync(0xffffffffu, w)) { if (!w) fail(ST_WAIT_MMA); ok = false; break; }
      }
      tc_fence_after();
      uint32_t s[SUB];
      tmem_ld32(tmem_s, s);
      tmem_ld32(tmem_s + 32, s + 32);
      tmem_wait_ld();
      if (n0 + SUB > full_upto || n0 < full_from) {
        // A band edge crosses these keys: this row sees columns [lo_rel, hi_rel).
        const int hi_rel = lim - n0, lo_rel = lo - n0;
        const int hi_min = __reduce_min_sync(0xffffffffu, hi_rel), lo_max = __reduce_max_sync(0xffffffffu, lo_rel);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (32 * c + 32 > hi_min) {
#pragma unroll
            for (int i = 32 * c; i < 32 * c + 32; ++i)
              if (i >= hi_rel) s[i] = 0xff800000u;  // -inf
          }
          if (32 * c < lo_max) {
#pragma unroll
            for (int i = 32 * c; i < 32 * c + 32; ++i)
              if (i < lo_rel) s[i] = 0xff800000u;
          }
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int i = 0; i < SUB; i += 4) {
        asm("max.f32 %0, %0, %1, %2;" : "+f"(mx0) : "f"(__uint_as_float(s[i + 0])), "f"(__uint_as_float(s[i + 1])));
        asm("max.f32 %0, %0, %1, %2;" : "+f"(mx1) : "f"(__uint_as_float(s[i + 2])), "f"(__uint_as_float(s[i + 3])));
      }
      const float m_new = fmaxf(m_run, fmaxf(mx0, mx1));
      bool want = false;
      if (m_run == -INFINITY) {
        m_run = m_new;  // nothing accumulated yet for this row
        growth = (n0 & SUB) == 0 ? 0.f : RESCALE_THRESHOLD;  // (first half of 128 keys: the second may not exceed it)
      } else {
        want = (m_new - m_run) * qk_scale > growth;
        growth = RESCALE_THRESHOLD;
      }
      if (__any_sync(0xffffffffu, want)) {
        // (S of this step certifies that the previous step's P V has completed)
        const float alpha = want ? fast_exp2((m_run - m_new) * qk_scale) : 1.0f;
        if (want) m_run = m_new;
        l_run *= alpha;
#pragma unroll
        for (int c = 0; c < D; c += 8) {
          uint32_t o[8];
          tmem_ld8(tmem_o + c, o);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st8(tmem_o + c, o);
        }
      }
      const float m_eff = (m_run == -INFINITY) ? 0.f : m_run;
      const float neg_ms = -m_eff * qk_scale;
      const uint64_t scale2 = f2_pack(qk_scale, qk_scale), neg_ms2 = f2_pack(neg_ms, neg_ms);
      uint64_t sum01 = 0ull, sum23 = 0ull;
#pragma unroll
      for (int i = 0; i < SUB; i += 4) {
        float p0, p1, p2, p3;
        const uint64_t x01 = f2_fma(f2_pack(__uint_as_float(s[i + 0]), __uint_as_float(s[i + 1])), scale2, neg_ms2);
        const uint64_t x23 = f2_fma(f2_pack(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])), scale2, neg_ms2);
        if ((PolyMask<D>::value >> ((i >> 1) & 7)) & 1u) {
          exp2_poly_pair(x01, p0, p1);
        } else {
          float x0, x1;
          f2_unpack(x01, x0, x1);
          p0 = fast_exp2(x0);
          p1 = fast_exp2(x1);
        }
        if ((PolyMask<D>::value >> (((i >> 1) + 1) & 7)) & 1u) {
          exp2_poly_pair(x23, p2, p3);
        } else {
          float x2, x3;
          f2_unpack(x23, x2, x3);
          p2 = fast_exp2(x2);
          p3 = fast_exp2(x3);
        }
        sum01 = f2_add(sum01, f2_pack(p0, p1));
        sum23 = f2_add(sum23, f2_pack(p2, p3));
        s[i / 2 + 0] = pack2<BF16>(p0, p1);
        s[i / 2 + 1] = pack2<BF16>(p2, p3);
        if constexpr (DROPOUT) {
          s[i / 2 + 0] &= keep_mask_pair(keep_bits[i >> 5], i & 31);
          s[i / 2 + 1] &= keep_mask_pair(keep_bits[i >> 5], (i & 31) + 2);
        }
      }
      tmem_st32(tmem_s, s);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
      float sum0, sum1, sum2, sum3;
      f2_unpack(sum01, sum0, sum1);
      f2_unpack(sum23, sum2, sum3);
      l_run += (sum0 + sum1) + (sum2 + sum3);
    }

    // ------------------------------------------------------------- epilogue
    if (ok && n_sub > 0) {
      const bool w = wait(o_full, 0);
      if (!__all_sync(0xffffffffu, w)) { if (!w) fail(ST_WAIT_MMA); ok = false; }
    }
    const bool empty = n_sub == 0 || m_run == -INFINITY || !(l_run > 0.f);
    if (ok && m_glob < args.M)
      args.lse[b * args.lse_stride_b + h * args.lse_stride_h + m_glob] = empty ? -INFINITY : m_run * args.sm_scale + logf(l_run);
    const int m_warp = m0 + warp * 32;  // first row of this warp's output box
    if (ok && m_warp < args.M) {
      // Scaled rows in the swizzled layout of the output tensor map, over the Q tile (its last reader has completed);
      // one TMA store of 32 rows per warp clips the rows past M.
      tc_fence_after();
      float inv = empty ? 0.f : 1.0f / l_run;
      if constexpr (DROPOUT) inv *= args.drop.inv_keep;
      const uint32_t row_addr = smem_u32(sQ) + row * Cfg::ROW_BYTES;
      const uint32_t swz = (row_addr >> 7) & (Cfg::ROW_BYTES / 16 - 1);
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t o[16];
        if (n_sub > 0) {
          tmem_ld16(tmem_o + c, o);
          tmem_wait_ld();
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = empty ? 0u : __float_as_uint(__uint_as_float(o[i]) * inv);
#pragma unroll
        for (int x = 0; x < 16; x += 8) {
          const uint32_t dst = row_addr + ((static_cast<uint32_t>((c + x) >> 3) ^ swz) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst),
                       "r"(pack2<BF16>(__uint_as_float(o[x + 0]), __uint_as_float(o[x + 1]))),
                       "r"(pack2<BF16>(__uint_as_float(o[x + 2]), __uint_as_float(o[x + 3]))),
                       "r"(pack2<BF16>(__uint_as_float(o[x + 4]), __uint_as_float(o[x + 5]))),
                       "r"(pack2<BF16>(__uint_as_float(o[x + 6]), __uint_as_float(o[x + 7])))
                       : "memory");
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        tma_store_4d(&tmO, sQ + warp * 32 * Cfg::ROW_BYTES, 0, m_warp, h, b);
        tma_store_commit();
        tma_store_wait_read();  // shared memory must outlive the read
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  __syncwarp();
  if (warp == 4) {
    if (*abort_flag) {
      // Give copies that may still be in flight time to land before shared memory is released.
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) {}
    }
    tmem_dealloc(tmem_base, Sm::TMEM_COLS);
  }
}

}  // namespace b200attn
