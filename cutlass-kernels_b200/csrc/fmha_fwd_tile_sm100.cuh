// Flash-attention forward for sm_100a with one 128-row query tile per CTA, for calls that have too few 256-row blocks for the
// SMs (fmha_fwd_sm100.cuh).  Stands where the reference has fmhaForwardPipelinedWspl (src/fmha-pipeline/fmha_pipe_ws.h:69-365).
//
//   warps 0-3   softmax and epilogue (thread r owns row r == TMEM lane r)
//   warp 4      UMMA issuer: S = Q K_j^T and O += P_j V_j, accumulators in TMEM
//   warp 5      TMA producer: Q once, then K_j, V_j tiles into a ring of shared-memory slots
//   warps 6-7   idle; they complete the second warpgroup so that registers can be moved from it (setmaxnreg)
//
// A CTA takes half an SM: 256 columns of tensor memory, at most 113 KB of shared memory, half the registers.  Two CTAs on an
// SM interleave as the two query tiles of the 256-row kernel do, but start and end on their own: the work comes in half the
// pieces, and the last wave in halves of SMs: 300 heads of 300 x 300, bf16 d = 128 causal: 48.4 -> 33.7 us.  K and V are read once
// per 128 rows instead of per 256, which is why long calls stay with the 256-row kernel.
//
// Where even the 128-row tiles are too few, a cluster of `splits` CTAs shares one: each takes a contiguous part of the key
// tiles; at the end every CTA leaves its unnormalised O (fp32) and each row's reference maximum and sum in its shared memory,
// and after a cluster barrier CTA c combines columns c * HD / splits .. through distributed shared memory, in rank order: 8
// heads, 512 x 4096: 51.2 -> 18.8 us (rule and more figures: capi.cu, tile_plan).
#pragma once
#include "fmha_softmax.cuh"

namespace cfk {

template <int DT, int PT, int HD>
struct FmhaTileCfg : FmhaCfg<DT, PT, HD> {
  using B = FmhaCfg<DT, PT, HD>;
  static constexpr int SMEM_HALF = 113 * 1024;             // two CTAs and the 1 KB each that the system reserves
  static constexpr int HEADB = 1024 + B::BARB + 4 * 128 * 4;   // alignment, barriers, row statistics of a split
  static constexpr int FIT = (SMEM_HALF - HEADB - B::TILEB) / B::SLOTB;
  static constexpr int NSLOT = FIT > 8 ? 8 : FIT;
  static_assert(NSLOT >= 2 && NSLOT * B::SLOTB >= 128 * HD * 4, "the ring holds O when the parts are merged");
  static constexpr int SMEM_BYTES = HEADB + B::TILEB + NSLOT * B::SLOTB;
  static constexpr int TMEM_COLS = 256, O_COL0 = 128, P_COL0 = 192;   // S [0, 128); O; d = 64: P in [192, 256)
  static constexpr int NTHREADS = 256;
  static constexpr int LAUNCH_REGS = 128, SOFTMAX_REGS = 208, AUX_REGS = 48;
  static_assert(128 * SOFTMAX_REGS + 128 * AUX_REGS <= NTHREADS * LAUNCH_REGS, "setmaxnreg would block forever");
};

template <int DT, int PT, int HD, int EMU>
__global__ void __launch_bounds__(256, 2)
fmha_fwd_tile_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                     const FmhaSplitParams sp) {
  using C = FmhaTileCfg<DT, PT, HD>;
  const FmhaParams& p = sp.p;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t sQ = smem_base;
  const uint32_t sRing = sQ + C::TILEB;
  const uint32_t sBar = sRing + C::NSLOT * C::SLOTB;
  const uint32_t sStat = sBar + C::BARB;                     // [3][128] floats: reference maximum (log2), sum, true maximum
  uint8_t* gBar = smem_gen + (sBar - smem_base);
  const uint32_t bar_q_full = sBar;
  const uint32_t bar_kv_full = sBar + 8;                     // [NSLOT]
  const uint32_t bar_kv_empty = bar_kv_full + 8 * C::NSLOT;  // [NSLOT]
  const uint32_t bar_s_full = bar_kv_empty + 8 * C::NSLOT;
  const uint32_t bar_p_full = bar_s_full + 8;                // [2] P of keys 0-63 / of keys 64-127
  const uint32_t bar_pv_done = bar_p_full + 16;              // d = 64: O += P V_j is complete
  const uint32_t bar_o_full = bar_pv_done + 8;
  const uint32_t bar_o_staged = bar_o_full + 8;
  const uint32_t off_misc = (bar_o_staged + 8) - sBar;
  static_assert(8 * (2 * C::NSLOT + 7) + 16 <= C::BARB, "barrier block overflows");
  volatile uint32_t* s_tmem_base = reinterpret_cast<volatile uint32_t*>(gBar + off_misc);
  volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(gBar + off_misc + 4);
  volatile uint32_t* s_skip = reinterpret_cast<volatile uint32_t*>(gBar + off_misc + 8);
  const AbortCtx actx{s_abort, p.status};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // Work item: p.nqblk counts 128-row query blocks here; the grouped, heaviest-first order of the other kernels.
  const int part = (int)blockIdx.x % sp.splits;
  int qblk, head, batch;
  {
    const int unit = (int)blockIdx.x / sp.splits;
    const int bh_total = p.B * p.H;
    const int per_group = p.group * p.nqblk;
    const int g = unit / per_group;
    const int rr = unit - g * per_group;
    const int left = bh_total - g * p.group;
    const int gsz = left < p.group ? left : p.group;
    qblk = p.nqblk - 1 - rr / gsz;
    const int bh = g * p.group + rr % gsz;
    batch = bh / p.H;
    head = bh - batch * p.H;
  }
  const int row0 = qblk * 128;
  const int diag_off = p.Skv - p.Sq;
  int n_all = (p.Skv + C::BN - 1) / C::BN;
  if (p.causal) {
    const int nc = (row0 + 127 + diag_off) / C::BN + 1;
    n_all = nc < n_all ? nc : n_all;
  }
  const int j0 = n_all * part / sp.splits;                   // this CTA's key tiles: j0 .. j0 + n_kv - 1
  const int n_kv = n_all * (part + 1) / sp.splits - j0;

  // Set-up as in fmha_fwd_sm100.cuh: ahead of the wait for the launch before, with Q and the first K on their way early.
  if (warp == 5 && lane == 0) {
    mbar_init(bar_q_full, 1);
    for (int i = 0; i < C::NSLOT; ++i) { mbar_init(bar_kv_full + 8 * i, 1); mbar_init(bar_kv_empty + 8 * i, 1); }
    mbar_init(bar_s_full, 1);
    mbar_init(bar_p_full, 4);
    mbar_init(bar_p_full + 8, 4);
    mbar_init(bar_pv_done, 1);
    mbar_init(bar_o_full, 1);
    mbar_init(bar_o_staged, 4);
    *s_abort = 0u;
    fence_barrier_init();
    fence_proxy_async_smem();
    grid_dependency_wait();
    if (n_kv > 0) {
      mbar_arrive_expect_tx(bar_q_full, C::TILEB);
      tma_load_5d(sQ, &tm_q, bar_q_full, 0, row0, 0, head, batch);
      mbar_arrive_expect_tx(bar_kv_full, C::TILEB);
      tma_load_5d(sRing, &tm_k, bar_kv_full, 0, j0 * C::BN, 0, head, batch);
    }
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_o);
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(s_tmem_base)), C::TMEM_COLS);
    tmem_relinquish();
    grid_dependency_launch();
  }
  if (warp == 5) __syncwarp();
  grid_dependency_wait();
  if (tid == 0) *s_skip = (uint32_t)(*reinterpret_cast<const volatile int*>(p.status) != 0);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *s_tmem_base;
  // A wait of an earlier launch gave up: nothing is computed and nothing written, but the CTAs of a cluster stay in step
  // (each read the status word for itself).
  const bool skip = *s_skip != 0u;

  bool split_p = false;   // bf16 only: few visible keys, P as hi + lo (lo in the upper half of the S columns)
  if constexpr (PT == kDtBF16) {
    int visible = p.Skv;     // of the first row of the 256-row block, so that both kernels decide, and round, alike
    if (p.causal) { const int v0 = (row0 & ~255) + diag_off + 1; visible = v0 < visible ? v0 : visible; }
    split_p = visible < p.split_keys;
  }
  const bool sep_p = C::SEP_P && !split_p;                   // P in a buffer of its own (see fmha_fwd_sm100.cuh)

  float m_ref = 0.f, m_true = -INFINITY, l = 0.f;
  bool ok = true;

  if (warp >= 4) {
    setmaxnreg_dec<C::AUX_REGS>();
    if (warp == 5) {
      // =========================== TMA producer: K_0 V_0 K_1 V_1 .. ===========================
      if (lane == 0 && n_kv > 0) {
        if (skip) {          // the two loads above must have landed before shared memory is given back
          mbar_wait(bar_q_full, 0, actx, kErrFmhaQFull);
          mbar_wait(bar_kv_full, 0, actx, kErrFmhaKvFull);
        } else {
          for (int idx = 1; idx < 2 * n_kv; ++idx) {
            const int slot = idx % C::NSLOT;
            const uint32_t ph = (idx / C::NSLOT) & 1;
            if (!mbar_wait(bar_kv_empty + 8 * slot, ph ^ 1u, actx, kErrFmhaKvEmpty)) break;
            const bool is_v = idx & 1;
            mbar_arrive_expect_tx(bar_kv_full + 8 * slot, is_v ? C::VTILEB : C::TILEB);
            tma_load_5d(sRing + slot * C::SLOTB, is_v ? &tm_v : &tm_k, bar_kv_full + 8 * slot, 0, (j0 + (idx >> 1)) * C::BN, 0,
                        head, batch);
          }
        }
      }
    } else if (warp == 4 && n_kv > 0 && !skip) {
      // =========================== UMMA issue (see fmha_fwd_sm100.cuh) ===========================
      const uint32_t leader = elect_one();
      const uint64_t aq0 = make_smem_desc(sQ, 16, C::SBO, C::SWZ);
      const uint64_t bk0 = make_smem_desc(sRing, 16, C::SBO, C::SWZ);
      const uint64_t bv0 = make_smem_desc(sRing, C::VSUBB, C::VSBO, C::VSWZ);
      const uint32_t tO = tmem_base + C::O_COL0;
      auto wait_slot = [&](int idx) -> bool {
        const bool r = mbar_wait_warp(bar_kv_full + 8 * (idx % C::NSLOT), (idx / C::NSLOT) & 1, actx, kErrFmhaKvFull);
        tc_fence_after_sync();
        return r;
      };
      auto issue_qk = [&](int idx) {
        const uint64_t b0 = desc_advance_lo(bk0, (idx % C::NSLOT) * C::SLOTB);
#pragma unroll
        for (int kk = 0; kk < C::QK_KSTEPS; ++kk) {
          const uint32_t off = (kk / C::KSPS) * C::SUBB + (kk % C::KSPS) * 32;
          umma_ss_e<C::KIND8, false>(tmem_base, desc_advance_lo(aq0, off), desc_advance_lo(b0, off), C::IDESC_QK,
                                     kk > 0 ? 1u : 0u, leader);
        }
        umma_commit_e<false>(bar_s_full, leader);
        umma_commit_e<false>(bar_kv_empty + 8 * (idx % C::NSLOT), leader);
      };
      // keys kk0 .. of the P at column `a` times V: steps k0 .. k0 + n - 1
      auto issue_pv = [&](uint32_t a, int idx, int k0, int n, uint32_t accumulate) {
        const uint64_t b0 = desc_advance_lo(bv0, (idx % C::NSLOT) * C::SLOTB);
#pragma unroll
        for (int k2 = 0; k2 < C::PV_KSTEPS; ++k2)
          if (k2 < n)
            umma_ts_e<C::KIND8_PV, false>(tO, a + (k0 + k2) * 8, desc_advance_lo(b0, (k0 + k2) * C::V_STEPB), C::IDESC_PV,
                                          k2 > 0 ? 1u : accumulate, leader);
      };
      ok = mbar_wait_warp(bar_q_full, 0, actx, kErrFmhaQFull) && wait_slot(0);
      if (ok) issue_qk(0);
      const uint32_t tP = tmem_base + (sep_p ? C::P_COL0 : 0);
      constexpr int HALF = C::PV_KSTEPS / 2;
      for (int j = 0; j < n_kv && ok; ++j) {
        const int vidx = 2 * j + 1, kidx = 2 * j + 2;
        const bool more = j + 1 < n_kv;
        const uint32_t acc = j > 0 ? 1u : 0u;
        if (!(ok = wait_slot(vidx))) break;
        if (!split_p) {      // with the two-term P the first-half barrier is not signalled
          if (!(ok = mbar_wait_warp(bar_p_full, j & 1, actx, kErrFmhaPFull))) break;
          tc_fence_after_sync();
          if (sep_p && more) {
            if (!(ok = wait_slot(kidx))) break;
            issue_qk(kidx);
          }
          issue_pv(tP, vidx, 0, HALF, acc);
        }
        if (!(ok = mbar_wait_warp(bar_p_full + 8, j & 1, actx, kErrFmhaPFull))) break;
        tc_fence_after_sync();
        if (split_p) {
          issue_pv(tP, vidx, 0, C::PV_KSTEPS, acc);
          if constexpr (PT == kDtBF16) issue_pv(tP + 64, vidx, 0, C::PV_KSTEPS, 1u);   // reads V at the same steps
        } else {
          issue_pv(tP, vidx, HALF, HALF, 1u);
        }
        if (sep_p) umma_commit_e<false>(bar_pv_done, leader);
        if (!more) umma_commit_e<false>(bar_o_full, leader);
        umma_commit_e<false>(bar_kv_empty + 8 * (vidx % C::NSLOT), leader);
        if (!sep_p && more) {
          if (!(ok = wait_slot(kidx))) break;
          issue_qk(kidx);
        }
      }
    }
    if (sp.splits > 1) {     // the two cluster barriers of the merge below
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    // =========================== softmax ===========================
    setmaxnreg_inc<C::SOFTMAX_REGS>();
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    const uint32_t tS = tmem_base + lane_base, tO = tS + C::O_COL0;
    const int row_g = row0 + tid;
    const int tile_min_lim = p.causal ? min(p.Skv - 1, row0 + diag_off) : p.Skv - 1;
    int lim = p.Skv - 1;
    if (p.causal) { const int cl = row_g + diag_off; lim = cl < lim ? cl : lim; }
    const float sl = p.scale_log2;
    uint32_t sreg[128];
    auto key_tile_loop = [&](auto split_c, auto own_c) {
      constexpr bool SPLIT = decltype(split_c)::value, OWN_P = decltype(own_c)::value;
      const uint32_t tP = OWN_P ? tS + C::P_COL0 : tS;
      for (int j = 0; j < n_kv; ++j) {
        ok = mbar_wait_warp(bar_s_full, j & 1, actx, kErrFmhaSFull);
        if (!ok) break;
        tc_fence_after_sync();
        tmem_ld_x32(tS + 0, sreg + 0);
        tmem_ld_x32(tS + 32, sreg + 32);
        tmem_ld_x32(tS + 64, sreg + 64);
        tmem_ld_x32(tS + 96, sreg + 96);
        uint32_t pv_seen = 0u;
        if (OWN_P && j > 0) pv_seen = mbar_test_wait(bar_pv_done, (uint32_t)(j - 1) & 1u);
        tmem_wait_ld();
        const int key0 = (j0 + j) * C::BN;
        ok = softmax_step<C, PT, HD, EMU, SPLIT>(sreg, tS, tP, tO, sl, j == 0, key0 + 127 > tile_min_lim, lim - key0, bar_p_full,
                                                 OWN_P ? bar_pv_done : 0u, (uint32_t)(j - 1) & 1u, pv_seen, actx, m_ref,
                                                 m_true, l);
        if (!ok) break;
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive_warp(bar_p_full + 8);
      }
    };
    if (!skip) {
      if constexpr (C::SEP_P) {
        if constexpr (PT == kDtBF16) {
          if (split_p) key_tile_loop(std::true_type{}, std::false_type{});
          else key_tile_loop(std::false_type{}, std::true_type{});
        } else {
          key_tile_loop(std::false_type{}, std::true_type{});
        }
      } else {
        if constexpr (PT == kDtBF16) {
          if (split_p) key_tile_loop(std::true_type{}, std::false_type{});
          else key_tile_loop(std::false_type{}, std::false_type{});
        } else {
          key_tile_loop(std::false_type{}, std::false_type{});
        }
      }
      if (n_kv > 0 && ok) {
        ok = mbar_wait_warp(bar_o_full, 0, actx, kErrFmhaOFull);
        tc_fence_after_sync();
      }
    }
    const float mref2 = m_ref * sl - C::PSHIFT;              // exponent origin of l, log2 domain
    if (sp.splits == 1) {
      // ---- output: normalise, stage over the drained ring, TMA store ----
      if (ok && !skip) {
        stage_output<C, HD>(tO, sRing, tid, p.out_scale / l, p.out_bf16 != 0);
        fence_proxy_async_smem();
        mbar_arrive_warp(bar_o_staged);
        if (tid == 0 && mbar_wait(bar_o_staged, 0, actx, kErrFmhaOStaged)) {
          tma_store_5d(&tm_o, sRing, 0, row0, 0, head, batch);
          tma_store_commit();
          tma_store_wait_read0();
        }
        if (row_g < p.Sq) {
          const size_t so = ((size_t)batch * p.H + head) * p.Sq + row_g;
          if (p.lse) p.lse[so] = 0.69314718055994531f * (mref2 + log2f(l));
          if (p.mi) p.mi[so] = m_true * sl;
          if (p.sprime) p.sprime[so] = l * exp2f(mref2 - m_true * sl);
        }
      }
    } else {
      // ---- this part's O and statistics to shared memory: [column / 4][row][16 bytes]; no visible key: maximum -inf ----
      if (ok && !skip && n_kv > 0) {
        uint32_t oreg[32];
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          tmem_ld_x32(tO + c * 32, oreg);
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < 8; ++g)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sRing + (c * 8 + g) * 2048 + tid * 16),
                         "r"(oreg[4 * g]), "r"(oreg[4 * g + 1]), "r"(oreg[4 * g + 2]), "r"(oreg[4 * g + 3]) : "memory");
        }
      }
      // No visible key, or none with a score above -inf.  The sum does not tell: masked keys add 2^-126 each where the
      // exponential is taken on the FMA pipe, against a reference maximum of 0.  A sum of NaN (NaN scores, which a maximum
      // passes over) is passed on.
      const bool none = n_kv == 0 || (m_true == -INFINITY && l == l);
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(sStat + tid * 4), "f"(none ? -INFINITY : mref2) : "memory");
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(sStat + 512 + tid * 4), "f"(none ? 0.f : l) : "memory");
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(sStat + 1024 + tid * 4), "f"(m_true * sl) : "memory");
      __syncwarp();
      cluster_sync_all();                                    // every part is in its CTA's shared memory
      if (!skip && !*s_abort && row_g < p.Sq) {
        float w[8], mx = -INFINITY, mt = -INFINITY, lsum = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          w[c] = c < sp.splits ? ld_shared_cluster_f32(map_to_cta(sStat + tid * 4, c)) : -INFINITY;
          mx = fmaxf(mx, w[c]);
        }
        // Parts that have left an O.  Those whose weight underflows to 0 count: NaN and infinite values reach the result.
        uint32_t has = 0u;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          if (w[c] != -INFINITY) has |= 1u << c;
          w[c] = w[c] == -INFINITY ? 0.f : ex2_approx(w[c] - mx);
          if (c < sp.splits) {
            lsum += w[c] * ld_shared_cluster_f32(map_to_cta(sStat + 512 + tid * 4, c));
            mt = fmaxf(mt, ld_shared_cluster_f32(map_to_cta(sStat + 1024 + tid * 4, c)));
          }
        }
        const float inv = p.out_scale / lsum;
        uint16_t* dst = reinterpret_cast<uint16_t*>(sp.o) + batch * sp.o_b + row_g * sp.o_s + head * sp.o_h;
        const int c4 = HD / 4 / sp.splits;                     // groups of four columns per CTA
        for (int g = part * c4; g < (part + 1) * c4; ++g) {
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if (has >> c & 1u) {                               // a part without a visible key has left no O
              const float4 v = ld_shared_cluster_f32x4(map_to_cta(sRing + g * 2048 + tid * 16, c));
              acc.x += w[c] * v.x; acc.y += w[c] * v.y; acc.z += w[c] * v.z; acc.w += w[c] * v.w;
            }
          }
          uint2 o2;
          o2.x = p.out_bf16 ? pack_bf16x2(acc.x * inv, acc.y * inv) : pack_f16x2(acc.x * inv, acc.y * inv);
          o2.y = p.out_bf16 ? pack_bf16x2(acc.z * inv, acc.w * inv) : pack_f16x2(acc.z * inv, acc.w * inv);
          *reinterpret_cast<uint2*>(dst + 4 * g) = o2;
        }
        if (part == 0) {
          const size_t so = ((size_t)batch * p.H + head) * p.Sq + row_g;
          if (p.lse) p.lse[so] = 0.69314718055994531f * (mx + log2f(lsum));
          if (p.mi) p.mi[so] = mt;
          if (p.sprime) p.sprime[so] = lsum * exp2f(mx - mt);
        }
      }
      __syncwarp();
      cluster_sync_all();                                    // the peers may still be reading this CTA's shared memory
    }
  }

  // ---- tear-down ----
  settle_if_aborted(s_abort);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

}  // namespace cfk
