// Attention of a few query rows against a long cache: O = softmax(Q K^T * scale) V, 16 query rows of a (batch, head) at a
// time.  The reference has no kernel of its own for this; it runs its prefill kernels (fmha_pipe_ws.h:69-365).
//
// What bounds it is reading K and V once.  The 256-row kernel (fmha_fwd_sm100.cuh) spends a chain of about 1.5 us per 128
// keys on rows that are nearly all padding, on one SM per (batch, head).  Here a (batch, head) is cut along its keys into
// as many CTAs as it takes to keep every SM loading, each a ring of TMA loads that is consumed by warp-level MMAs:
//
//   warps 0-3   each takes a quarter of the keys of every tile: S = Q K^T, online softmax, O += P V, all in registers
//   warp 4      TMA producer: tiles of 64 or 128 keys, K and V on one barrier, into a ring of shared-memory slots
//
// A query tile of 16 rows is what mma.sync.m16n8k16 takes; a tcgen05.mma has at least 64 rows, and its way through tensor
// memory costs more than the arithmetic, which needs a fraction of the time the bytes take.  One row against 6001 keys, 128
// heads, d = 128, bf16 (393 MB): 61 us, 6.4 TB/s, against 70.6 in the 256-row kernel with the same launches; d = 64: 35.1
// against 57.7; e4m3: 36.5 against 61.4; 2 heads x 65536 keys: 57.5 against 679 (the rule and more figures: capi.cu,
// decode_is_faster).  Every warp keeps a maximum, a sum
// and an output of its own, so nothing synchronises inside the loop; at the end the four are merged through shared memory and
// the CTAs of one (batch, head), which form a cluster, through distributed shared memory.  So there is no workspace in global
// memory, no second launch, and calls on several streams share nothing.
// e4m3 operands are widened to fp16 (exact) in registers and P is kept in fp16; bf16 follows the two-term rule of the
// prefill kernels (FmhaParams::split_keys).
#pragma once
#include "fmha_softmax.cuh"

namespace cfk {

template <int DT, int PT, int HD>
struct DecodeCfg {
  static constexpr int ESZ = (DT == kDtE4M3) ? 1 : 2, PESZ = (PT == kDtE4M3) ? 1 : 2;
  static constexpr int ROWS = 16, NWARP = 4;
  // Keys per tile: a round of the producer (wait for the slot, announce the bytes, issue the copies) takes the same time however
  // small the tile is, so short rows travel 128 at a time: d = 64, 16 bit, one CTA, 65536 keys as 2048 copies of 64 keys with a
  // barrier each: 322 us, 0.16 per round.
  static constexpr int ROWB = HD * ESZ, SPANB = ROWB < 128 ? ROWB : 128;
  static constexpr int VROWB = HD * PESZ, VSPANB = VROWB < 128 ? VROWB : 128;
  static constexpr int TN = decode_tile_keys(HD, PESZ), NK = TN / NWARP, NT = NK / 8;   // keys and 8-key columns per warp
  static constexpr int QTILEB = ROWS * ROWB, KTILEB = TN * ROWB, VTILEB = TN * VROWB;
  static constexpr int SLOTB = KTILEB + VTILEB;
  static constexpr int MAXSLOT = 12;
  static constexpr int CTAS = decode_ctas_per_sm(HD, ESZ, PESZ);
  static constexpr int QSTEPS = HD / 16;
  static constexpr bool Q_REGS = HD < 128;         // Q fragments in registers, else in shared memory in fragment order
  static constexpr int QFRAGB = Q_REGS ? 0 : QSTEPS * 512;
  static constexpr int MISCB = 16 * MAXSLOT + 16 + 2 * 4 * (NWARP + 1) * ROWS;
  static constexpr int HEADB = (QTILEB + QFRAGB + MISCB + 1023) / 1024 * 1024;   // everything but the ring
  // Slots of the ring: what the CTAs that share an SM leave room for, and no more than a CTA has tiles, so that short calls
  // get more CTAs per SM.  The ring also holds the outputs of the warps when they are merged.
  static int slots(long long ctas, int sms, int tiles_per_cta) {
    const int want = ctas <= sms ? 1 : (ctas <= 2LL * sms ? 2 : 3), per_sm = want < CTAS ? want : CTAS;
    const int fit = ((per_sm == 1 ? 224 : per_sm == 2 ? 111 : 73) * 1024 - HEADB) / SLOTB;
    int n = fit < 1 ? 1 : (fit > MAXSLOT ? MAXSLOT : fit);
    return tiles_per_cta < n ? tiles_per_cta : n;
  }
  static int smem_bytes(int nslot, int rows) {
    const int merge = NWARP * (rows < ROWS ? rows : ROWS) * HD * 4, ring = nslot * SLOTB;
    return 1024 + HEADB + (ring > merge ? ring : merge);
  }
  static constexpr int SMEM_MAX = 227 * 1024;
  static constexpr int NTHREADS = 32 * (NWARP + 1);
};

// Volatile keeps these behind the barrier wait that says the tile has landed; the MMAs between them may be scheduled freely.
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  if constexpr (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};" : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};" : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four e4m3 values of a word -> two packed fp16 pairs (exact)
__device__ __forceinline__ void widen_e4m3(uint32_t w, uint32_t& lo, uint32_t& hi) {
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, a;\n\tcvt.rn.f16x2.e4m3x2 %1, b;\n\t}"
      : "=r"(lo), "=r"(hi) : "r"(w));
}
// Byte offset of 16-byte piece `even + bit` of row `row` in a tile of ROWS rows as the tensor maps lay it out: spans of
// SPANB bytes one after the other, the pieces of a row permuted by the 128- or 64-byte swizzle.  `even` is a constant at
// every use, so that a step costs one exclusive-or.
template <int ROWS, int SPANB>
__device__ __forceinline__ uint32_t tile_piece(int row, int even, int bit) {
  constexpr int CPS = SPANB / 16;
  const int x = SPANB == 128 ? (row & 7) : ((row >> 1) & 3);
  return (uint32_t)((even / CPS) * (ROWS * SPANB) + row * SPANB + (((even % CPS) << 4) ^ ((bit ^ x) << 4)));
}
template <int DT, int PT, int HD>
__global__ void __launch_bounds__(160, (DecodeCfg<DT, PT, HD>::CTAS))
fmha_decode_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const FmhaSplitParams dp) {
  using C = DecodeCfg<DT, PT, HD>;
  constexpr bool BF16 = PT == kDtBF16;
  const FmhaParams& p = dp.p;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t sQ = smem_base, sQf = sQ + C::QTILEB, sBar = sQf + C::QFRAGB;
  const uint32_t sRing = smem_base + C::HEADB;                // dp.nslot slots
  const uint32_t bar_full = sBar, bar_empty = sBar + 8 * C::MAXSLOT, bar_q = sBar + 16 * C::MAXSLOT;
  uint8_t* gMisc = smem_gen + (bar_q + 8 - smem_base);
  volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(gMisc);
  volatile uint32_t* s_skip = reinterpret_cast<volatile uint32_t*>(gMisc + 4);
  float* s_m = reinterpret_cast<float*>(gMisc + 8);           // [NWARP + 1][16]: row maxima of the warps, of the CTA
  float* s_l = s_m + (C::NWARP + 1) * C::ROWS;                // [NWARP + 1][16]: row sums
  float* s_o = reinterpret_cast<float*>(smem_gen + C::HEADB);  // [NWARP][rows][HD], over the ring once it is drained
  const AbortCtx actx{s_abort, p.status};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)blockIdx.x % dp.splits, unit = (int)blockIdx.x / dp.splits;
  const int qb = unit % dp.nqb, bh = unit / dp.nqb;
  const int batch = bh / p.H, head = bh - batch * p.H;
  const int row0 = dp.row_first + qb * C::ROWS;
  const int nrows = min(C::ROWS, p.Sq - row0);
  const int diag_off = p.Skv - p.Sq;
  const int visible = p.causal ? min(p.Skv, row0 + nrows + diag_off) : p.Skv;   // keys the last row sees
  const int ntiles = (visible + C::TN - 1) / C::TN;
  const int t0 = (int)((long long)ntiles * rank / dp.splits), t1 = (int)((long long)ntiles * (rank + 1) / dp.splits);

  auto load = [&](int slot, int j) {                          // K and V of tile j
    mbar_arrive_expect_tx(bar_full + 8 * slot, C::SLOTB);
    tma_load_5d(sRing + slot * C::SLOTB, &tm_k, bar_full + 8 * slot, 0, j * C::TN, 0, head, batch);
    tma_load_5d(sRing + slot * C::SLOTB + C::KTILEB, &tm_v, bar_full + 8 * slot, 0, j * C::TN, 0, head, batch);
  };
  const int early = min(t1 - t0, dp.nslot);                   // loads that need no free slot: issued in the set-up

  grid_dependency_launch();
  if (warp == C::NWARP && lane == 0) {
    for (int i = 0; i < dp.nslot; ++i) { mbar_init(bar_full + 8 * i, 1); mbar_init(bar_empty + 8 * i, C::NWARP); }
    mbar_init(bar_q, 1);
    *s_abort = 0u;
    fence_barrier_init();
    fence_proxy_async_smem();
    grid_dependency_wait();
    mbar_arrive_expect_tx(bar_q, C::QTILEB);
    tma_load_5d(sQ, &tm_q, bar_q, 0, row0, 0, head, batch);
    for (int i = 0; i < early; ++i) load(i, t0 + i);
  }
  if (warp == C::NWARP) __syncwarp();
  grid_dependency_wait();
  if (tid == 0) *s_skip = (uint32_t)(*reinterpret_cast<const volatile int*>(p.status) != 0);
  __syncthreads();
  const bool skip = *s_skip != 0u;                            // a wait of an earlier launch gave up: write nothing

  const float sl = p.scale_log2;
  float o[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) o[i][k] = 0.f;
  float m_true[2] = {-INFINITY, -INFINITY};
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};     // rows lane / 4 and lane / 4 + 8

  if (warp == C::NWARP) {
    if (lane == 0) {
      bool ok = true;
      if (skip) {                                             // what is on its way must land before the CTA ends
        ok = mbar_wait(bar_q, 0, actx, kErrDecodeFull);
        for (int i = 0; i < early && ok; ++i) ok = mbar_wait(bar_full + 8 * i, 0, actx, kErrDecodeFull);
      } else {
        int slot = 0;
        uint32_t phase = 0;                                   // of the first use of the ring, which has just begun
        for (int j = t0 + early; j < t1; ++j) {
          if (!mbar_wait(bar_empty + 8 * slot, phase, actx, kErrDecodeEmpty)) break;
          load(slot, j);
          if (++slot == dp.nslot) { slot = 0; phase ^= 1u; }
        }
      }
    }
  } else if (!skip) {
    bool ok = mbar_wait_warp(bar_q, 0, actx, kErrDecodeFull);
    // ---- Q fragments (A operand, 16 rows x 16 per step) ----
    [[maybe_unused]] uint32_t qf[C::Q_REGS ? C::QSTEPS : 1][4];
    const int a_row = (lane & 7) + ((lane >> 3) & 1) * 8;
    auto load_q = [&](int s, uint32_t (&f)[4]) {
      if constexpr (C::ESZ == 2) {
        ldsm_x4(f, sQ + tile_piece<C::ROWS, C::SPANB>(a_row, 2 * s, lane >> 4));
      } else {   // a 16-byte piece is a whole step; positions 2t, 2t+1 / 2t+8, 2t+9 of it are elements 4t .. 4t+3
        uint32_t w[4];
        ldsm_x4(w, sQ + tile_piece<C::ROWS, C::SPANB>(a_row, s & ~1, lane >> 4));
        widen_e4m3(w[(s & 1) * 2], f[0], f[2]);
        widen_e4m3(w[(s & 1) * 2 + 1], f[1], f[3]);
      }
    };
    if (ok) {
      if constexpr (C::Q_REGS) {
#pragma unroll
        for (int s = 0; s < C::QSTEPS; ++s) load_q(s, qf[s]);
      } else {
        for (int s = warp; s < C::QSTEPS; s += C::NWARP) {
          uint32_t f[4];
          if constexpr (C::ESZ == 2) load_q(s, f);
          else { if (s & 1) load_q(1 + (s & ~1), f); else load_q(s & ~1, f); }
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sQf + s * 512 + lane * 16), "r"(f[0]), "r"(f[1]),
                       "r"(f[2]), "r"(f[3]) : "memory");
        }
      }
    }
    if constexpr (!C::Q_REGS) named_bar_sync(1, 32 * C::NWARP);

    const int lim0 = p.causal ? min(p.Skv - 1, row0 + (lane >> 2) + diag_off) : p.Skv - 1;        // last visible key
    const int lim1 = p.causal ? min(p.Skv - 1, row0 + (lane >> 2) + 8 + diag_off) : p.Skv - 1;
    const int min_lim = p.causal ? min(p.Skv - 1, row0 + diag_off) : p.Skv - 1;
    bool split = false;
    if constexpr (BF16) {   // by the first row of the 256-row block (d = 256: 128), as in the kernels that take such blocks
      const int first = row0 & ~(HD == 256 ? 127 : 255);
      split = (p.causal ? min(p.Skv, first + diag_off + 1) : p.Skv) < p.split_keys;
    }
    const int k16 = warp * C::NK;                                // this warp's keys within a tile
    const int kb_row = k16 + (lane & 7) + (C::ESZ == 2 ? ((lane >> 4) & 1) : ((lane >> 3) & 1)) * 8;
    const int kb_chunk = C::ESZ == 2 ? (lane >> 3) & 1 : lane >> 4;
    const int v_row = k16 + (lane & 7) + ((lane >> 3) & 1) * 8;

    int slot = 0;
    uint32_t phase = 0;                                        // of the ring at `slot`
    float mt[2] = {-INFINITY, -INFINITY};                      // largest score this thread has seen (m may lag behind)
    for (int j = t0; j < t1; ++j) {
      ok = mbar_wait_warp(bar_full + 8 * slot, phase, actx, kErrDecodeFull);
      if (!ok) break;
      // ---- S = Q K^T: keys k16 + 8 n .. + 7 in s[n]; with two columns, odd steps have sums of their own (shorter chains) ----
      constexpr int NS = C::NT == 2 ? 4 : C::NT;
      float s[NS][4];
#pragma unroll
      for (int n = 0; n < NS; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
      const uint32_t kt = sRing + slot * C::SLOTB;
      auto q_frag = [&](int st, uint32_t (&a)[4]) {
        if constexpr (C::Q_REGS) {
#pragma unroll
          for (int x = 0; x < 4; ++x) a[x] = qf[C::Q_REGS ? st : 0][x];
        } else {
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                       : "r"(sQf + st * 512 + lane * 16));
        }
      };
#pragma unroll
      for (int st = 0; st < C::QSTEPS; st += 2) {
        uint32_t a[4], a2[4];
        q_frag(st, a);
        q_frag(st + 1, a2);
#pragma unroll
        for (int n = 0; n < C::NT; n += 2) {
          constexpr int X = C::NT == 2 ? 2 : 0;                // where odd steps are summed
          uint32_t b[4];
          if constexpr (C::ESZ == 2) {
            uint32_t b2[4];
            ldsm_x4(b, kt + tile_piece<C::TN, C::SPANB>(kb_row, 2 * st, kb_chunk) + n * 8 * C::SPANB);
            ldsm_x4(b2, kt + tile_piece<C::TN, C::SPANB>(kb_row, 2 * st + 2, kb_chunk) + n * 8 * C::SPANB);
            mma_16816<DT == kDtBF16>(s[n], a[0], a[1], a[2], a[3], b[0], b[1]);
            mma_16816<DT == kDtBF16>(s[n + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
            mma_16816<DT == kDtBF16>(s[n + X], a2[0], a2[1], a2[2], a2[3], b2[0], b2[1]);
            mma_16816<DT == kDtBF16>(s[n + 1 + X], a2[0], a2[1], a2[2], a2[3], b2[2], b2[3]);
          } else {
            uint32_t b0, b1;
            ldsm_x4(b, kt + tile_piece<C::TN, C::SPANB>(kb_row, st, kb_chunk) + n * 8 * C::SPANB);
            widen_e4m3(b[0], b0, b1);
            mma_16816<false>(s[n], a[0], a[1], a[2], a[3], b0, b1);
            widen_e4m3(b[1], b0, b1);
            mma_16816<false>(s[n + 1], a[0], a[1], a[2], a[3], b0, b1);
            widen_e4m3(b[2], b0, b1);
            mma_16816<false>(s[n + X], a2[0], a2[1], a2[2], a2[3], b0, b1);
            widen_e4m3(b[3], b0, b1);
            mma_16816<false>(s[n + 1 + X], a2[0], a2[1], a2[2], a2[3], b0, b1);
          }
        }
      }
      if constexpr (C::NT == 2) {
#pragma unroll
        for (int e = 0; e < 4; ++e) { s[0][e] += s[2][e]; s[1][e] += s[3][e]; }
      }

      // ---- online softmax; a thread has rows lane/4 (+8) and of every 8 keys 2 (lane%4) and the next ----
      const int key0 = j * C::TN + k16;
      if (key0 + C::NK - 1 > min_lim) {
        const int c = key0 + (lane & 3) * 2;
#pragma unroll
        for (int n = 0; n < C::NT; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (c + 8 * n + e > lim0) s[n][e] = -INFINITY;
            if (c + 8 * n + e > lim1) s[n][2 + e] = -INFINITY;
          }
      }
      bool move = false;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float mx = fmaxf(s[0][2 * r], s[0][2 * r + 1]);
#pragma unroll
        for (int n = 1; n < C::NT; ++n) mx = max3(mx, s[n][2 * r], s[n][2 * r + 1]);
        mt[r] = fmaxf(mt[r], mx);
        move = move || (mx - m[r]) * sl > 8.f;                 // m lags by at most 2^8, as in prefill
      }
      if (__any_sync(0xffffffffu, move)) {
        float f[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float mn = mt[r];                                    // the row's largest score so far, over its four threads
          mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
          mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
          f[r] = mn == m[r] ? 1.f : ex2_approx((m[r] - mn) * sl);
          m[r] = mn;
          l[r] *= f[r];
        }
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) { o[n][0] *= f[0]; o[n][1] *= f[0]; o[n][2] *= f[1]; o[n][3] *= f[1]; }
      }
      uint32_t pa[C::NT / 2][4];                               // P as the A operand: a0, a1: keys 0-7, rows / rows + 8; ..
      [[maybe_unused]] uint32_t pl[C::NT / 2][4];
      const float negm[2] = {m[0] == -INFINITY ? 0.f : -m[0] * sl, m[1] == -INFINITY ? 0.f : -m[1] * sl};
#pragma unroll
      for (int n = 0; n < C::NT; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float u = ex2_approx(fmaf(s[n][2 * r], sl, negm[r])), v = ex2_approx(fmaf(s[n][2 * r + 1], sl, negm[r]));
          l[r] += u + v;
          uint32_t& w = pa[n >> 1][2 * (n & 1) + r];
          w = BF16 ? pack_bf16x2(u, v) : pack_f16x2(u, v);
          if constexpr (BF16)
            pl[n >> 1][2 * (n & 1) + r] = pack_bf16x2(u - __uint_as_float(w << 16), v - __uint_as_float(w & 0xffff0000u));
        }

      // ---- O += P V ----
      const uint32_t vt = kt + C::KTILEB;
      auto pv = [&](const uint32_t (&a)[4], int g) {           // keys k16 + 16 g .. + 15
#pragma unroll
        for (int c = 0; c < C::VROWB / 16; c += 2) {
          uint32_t b[4];
          ldsm_x4_t(b, vt + tile_piece<C::TN, C::VSPANB>(v_row, c, lane >> 4) + g * 16 * C::VSPANB);
          if constexpr (C::PESZ == 2) {
            mma_16816<BF16>(o[c], a[0], a[1], a[2], a[3], b[0], b[1]);
            mma_16816<BF16>(o[c + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
          } else {
            // a word holds elements 2g, 2g+1 (d) of keys 2t and 2t+1: widened and regrouped by d, piece c gives the even
            // d of its 16 in o[2c] and the odd ones in o[2c + 1]
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              uint32_t k0, k1, k8, k9;
              widen_e4m3(b[2 * x], k0, k1);
              widen_e4m3(b[2 * x + 1], k8, k9);
              mma_16816<false>(o[2 * (c + x)], a[0], a[1], a[2], a[3], __byte_perm(k0, k1, 0x5410), __byte_perm(k8, k9, 0x5410));
              mma_16816<false>(o[2 * (c + x) + 1], a[0], a[1], a[2], a[3], __byte_perm(k0, k1, 0x7632),
                               __byte_perm(k8, k9, 0x7632));
            }
          }
        }
      };
#pragma unroll
      for (int g = 0; g < C::NT / 2; ++g) {
        pv(pa[g], g);
        if constexpr (BF16)
          if (split) pv(pl[g], g);
      }
      mbar_arrive_warp(bar_empty + 8 * slot);
      if (++slot == dp.nslot) { slot = 0; phase ^= 1u; }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {                              // the true maximum, for FmhaParams::mi and sprime
      mt[r] = fmaxf(mt[r], __shfl_xor_sync(0xffffffffu, mt[r], 1));
      m_true[r] = fmaxf(mt[r], __shfl_xor_sync(0xffffffffu, mt[r], 2));
    }
  }

  // ---- merge of the four warps: maxima and sums first, then the outputs at the CTA's maximum ----
  settle_if_aborted(s_abort);
  __syncthreads();                                             // the ring is drained
  if (warp < C::NWARP) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
      if (m_true[r] != m[r]) l[r] *= ex2_approx((m[r] - m_true[r]) * sl);
      if ((lane & 3) == 0) {
        s_m[warp * C::ROWS + (lane >> 2) + 8 * r] = m_true[r];
        s_l[warp * C::ROWS + (lane >> 2) + 8 * r] = l[r];
      }
    }
  }
  __syncthreads();
  if (warp < C::NWARP) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = (lane >> 2) + 8 * r;
      float mc = s_m[row];
#pragma unroll
      for (int w = 1; w < C::NWARP; ++w) mc = fmaxf(mc, s_m[w * C::ROWS + row]);
      const float base = mc == -INFINITY ? 0.f : mc;
      if (warp == 0 && (lane & 3) == 0) {
        float lc = 0.f;
#pragma unroll
        for (int w = 0; w < C::NWARP; ++w) lc += s_l[w * C::ROWS + row] * ex2_approx((s_m[w * C::ROWS + row] - base) * sl);
        s_m[C::NWARP * C::ROWS + row] = mc;
        s_l[C::NWARP * C::ROWS + row] = lc;
      }
      if (row < nrows) {
        const float f = ex2_approx((m[r] - base) * sl);
        float* dst = s_o + (warp * nrows + row) * HD;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) {
          if constexpr (C::PESZ == 2) {
            *reinterpret_cast<float2*>(dst + n * 8 + (lane & 3) * 2) = make_float2(o[n][2 * r] * f, o[n][2 * r + 1] * f);
          } else {
            dst[(n >> 1) * 16 + (lane & 3) * 4 + (n & 1)] = o[n][2 * r] * f;
            dst[(n >> 1) * 16 + (lane & 3) * 4 + 2 + (n & 1)] = o[n][2 * r + 1] * f;
          }
        }
      }
    }
  }
  __syncthreads();
  const int items = nrows * (HD / 4);                          // four outputs each
  float4* o4 = reinterpret_cast<float4*>(s_o);
  for (int e = tid; e < items; e += C::NTHREADS) {
    float4 a = o4[e];
#pragma unroll
    for (int w = 1; w < C::NWARP; ++w) {
      const float4 b = o4[w * items + e];
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    o4[e] = a;
  }

  // ---- merge of the cluster: CTA `rank` writes its share of the elements ----
  if (dp.splits > 1) cluster_sync_all(); else __syncthreads();
  const uint32_t sM = smem_u32(s_m + C::NWARP * C::ROWS), sL = smem_u32(s_l + C::NWARP * C::ROWS), sO = sRing;
  if (!skip) {
    const int e0 = items * rank / dp.splits, e1 = items * (rank + 1) / dp.splits;
    for (int e = e0 + tid; e < e1; e += C::NTHREADS) {
      const int row = e / (HD / 4), col = (e % (HD / 4)) * 4;
      float mt = -INFINITY, lt = 0.f;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int c = 0; c < dp.splits; ++c) mt = fmaxf(mt, ld_shared_cluster_f32(map_to_cta(sM + row * 4, c)));
      const float base = mt == -INFINITY ? 0.f : mt;
      for (int c = 0; c < dp.splits; ++c) {
        const float f = ex2_approx((ld_shared_cluster_f32(map_to_cta(sM + row * 4, c)) - base) * sl);
        lt += f * ld_shared_cluster_f32(map_to_cta(sL + row * 4, c));
        const float4 v = ld_shared_cluster_f32x4(map_to_cta(sO + e * 16, c));
        acc.x += f * v.x; acc.y += f * v.y; acc.z += f * v.z; acc.w += f * v.w;
      }
      const float inv = p.out_scale / lt;
      uint2 w;
      w.x = p.out_bf16 ? pack_bf16x2(acc.x * inv, acc.y * inv) : pack_f16x2(acc.x * inv, acc.y * inv);
      w.y = p.out_bf16 ? pack_bf16x2(acc.z * inv, acc.w * inv) : pack_f16x2(acc.z * inv, acc.w * inv);
      uint16_t* dst = reinterpret_cast<uint16_t*>(dp.o) + batch * dp.o_b + (row0 + row) * dp.o_s + head * dp.o_h + col;
      *reinterpret_cast<uint2*>(dst) = w;
      if (col == 0) {
        const size_t so = ((size_t)batch * p.H + head) * p.Sq + row0 + row;
        if (p.lse) p.lse[so] = 0.69314718055994531f * (base * sl + log2f(lt));
        if (p.mi) p.mi[so] = mt * sl;
        if (p.sprime) p.sprime[so] = lt;
      }
    }
  }
  if (dp.splits > 1) cluster_sync_all();                       // the peers may still be reading this CTA's shared memory
}

}  // namespace cfk
