// Dense GEMM for sm_100a:  D[r][c] = alpha * sum_k X[r][k] * Y[c][k] + beta * D[r][c], X and Y
// K-contiguous, D row-major with leading dimension ldd, fp32 accumulation in tensor memory.
// It stands where the reference has gemm<> / gemm_device (src/cute-gemm-tma-gma/gemm.cu:336-463,
// 57-334): that kernel is a single-stage TMA -> WGMMA loop that stores register accumulators straight
// to global memory, ignores alpha / beta and accumulates in the output type.  Here a pair of CTAs on two
// SMs (tcgen05 cta_group::2) computes a tile of 256 rows x TN columns, TN = 256, 128 or 64:
//
//   warp 0     TMA producer: this CTA's 128 rows of X and its TN / 2 rows of Y per 64-wide k-block, into a
//              ring of 6 or 4 stages; both CTAs signal the same barrier in the leader (no multicast: each CTA
//              fetches only what its own SM consumes)
//   warp 1     UMMA issuer (leader CTA only): 256 x TN x 16 tcgen05.mma over the pair, two accumulator
//              buffers of TN TMEM columns per CTA
//   warps 2-5  epilogue: TMEM -> registers -> alpha/beta -> output type -> a swizzled staging tile in shared
//              memory (128 rows x 128 bytes, two of them) -> TMA store, overlapped with the next tile's main
//              loop.  (The reference writes its register accumulators to global memory thread by thread,
//              gemm.cu:329-331.)
//
// The pair halves the B-operand bytes each SM reads from shared memory per FLOP, which is what bounds a
// single-CTA 128 x 256 tile.  Pairs are persistent (one per two SMs) and walk the tile list in bands of
// 8 row-tiles so that concurrently running tiles share X and Y panels in L2.  The reference's column-major
// C (gemm.cu:388-389) is the row-major D of the swapped problem (X = B, Y = A), so one kernel serves both
// output orders.
//
// Where the tiles of D are too few for the SMs, `splits` pairs share one tile: a cluster of 2 * splits CTAs, each pair with a
// part of the reduction.  At the end every CTA leaves its fp32 accumulator, except the columns it is going to finish itself,
// in its shared memory (the ring is free by then); after a cluster barrier it adds the other pairs' parts of its columns
// through distributed shared memory, in pair order, and writes them.  No workspace, and the result does not depend on timing.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <utility>

#include "common.cuh"
#include "host_util.h"

namespace cfk {

constexpr int kErrGemmFull = 201, kErrGemmEmpty = 202, kErrGemmAccFull = 203, kErrGemmAccEmpty = 204,
              kErrGemmStaged = 205, kErrGemmStageFree = 206;

struct GemmParams {
  int R, Cn, K, L;       // rows of X / D, rows of Y (= columns of D), reduction length, batch count
  int64_t ldd;           // leading dimension of D (elements)
  int64_t d_batch;       // elements between consecutive D matrices
  void* d;
  const void* src;       // matrix of the beta term (same layout as D); D itself when the update is in place
  float alpha, beta;
  int bf16;
  int tf32;              // operands and D are fp32; the tensor core runs them as tf32 (kind::tf32, 8 elements per k-step)
  int tiles_r, tiles_c;  // tiles of 256 x TN
  int splits;            // pairs that share a tile, each with a part of the reduction
  int direct;            // one cluster per tile, which writes D from registers (with a split, or with `trans`)
  int trans;             // X holds the columns of D and Y its rows: D[c][r], still with leading dimension ldd
  int* status;
};

template <int TN_>
struct GemmCfg {
  static constexpr int TM = 256, TN = TN_;                    // tile of the CTA pair
  static constexpr int BM = 128, BNH = TN / 2, BK = 64;       // per CTA: rows of X, rows of Y, k extent
  // k-blocks per stage: a 256-wide tile hides a round of the producer and of the UMMA warp (barrier wait, announced bytes,
  // commit) behind 512 clk of MMA per k-block; a narrower one has 256 or 128 clk and shares a round between two k-blocks
  // (0.17 and 0.15 us per k-block as measured, where 512 clk take 0.30).
  static constexpr int KSUB = TN == 256 ? 1 : 2;
  static constexpr int XSUB = BM * BK * 2, YSUB = BNH * BK * 2;           // bytes per k-block
  static constexpr int XB = KSUB * XSUB, YB = KSUB * YSUB;                // bytes per stage
  static constexpr int NSTAGE = TN == 256 ? 6 : 4;
  static constexpr int STAGEB = 128 * 128;                    // output staging tile: 128 rows x 128 bytes
  static constexpr int SMEM_BYTES = 1024 + NSTAGE * (XB + YB) + 2 * STAGEB + 256;
  static constexpr int NTHREADS = 192;
  static constexpr int UNITS = TN / 32, UNITB = 128 * 32 * 4; // split: 32 columns of a CTA's accumulator in shared memory
  static_assert(UNITS * UNITB <= NSTAGE * (XB + YB), "split: the accumulator is handed over in the ring");
  static_assert(8 * (2 * NSTAGE + 8) + 8 <= 256, "barrier block overflows");
};
constexpr int kGemmBand = 8;

__device__ __forceinline__ void tile_coords(int tile, int tiles_r, int tiles_c, int& tr, int& tc, int& batch) {
  const int per_batch = tiles_r * tiles_c;
  batch = tile / per_batch;
  int t = tile - batch * per_batch;
  const int band_tiles = kGemmBand * tiles_c;
  const int band = t / band_tiles;
  const int first_r = band * kGemmBand;
  const int rows_in_band = (tiles_r - first_r) < kGemmBand ? (tiles_r - first_r) : kGemmBand;
  t -= band * band_tiles;
  tr = first_r + t % rows_in_band;
  tc = t / rows_in_band;
  if (band & 1) tc = tiles_c - 1 - tc;   // back and forth: a band starts on the Y panels the band before it ended on
}

// The beta term.  32 columns of a row of the source matrix, from element `at` on, `cols` of which exist, are read ahead of
// their use: a read takes about a microsecond, and the epilogue would otherwise wait for one per 32 columns.
struct SourceRow { uint4 x[8]; };     // 8 pieces of 4 fp32, or 4 of 8 16-bit values
__device__ __forceinline__ void load_source(SourceRow& s, const GemmParams& p, size_t at, int cols) {
  if (p.tf32) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(p.src) + at);
#pragma unroll
    for (int g = 0; g < 8; ++g) s.x[g] = g * 4 < cols ? src[g] : make_uint4(0u, 0u, 0u, 0u);
  } else {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.src) + at);
#pragma unroll
    for (int g = 0; g < 4; ++g) s.x[g] = g * 8 < cols ? src[g] : make_uint4(0u, 0u, 0u, 0u);
  }
}
__device__ __forceinline__ void add_source(float (&v)[32], const GemmParams& p, const SourceRow& s) {
  if (p.tf32) {
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      v[g * 4] += p.beta * __uint_as_float(s.x[g].x); v[g * 4 + 1] += p.beta * __uint_as_float(s.x[g].y);
      v[g * 4 + 2] += p.beta * __uint_as_float(s.x[g].z); v[g * 4 + 3] += p.beta * __uint_as_float(s.x[g].w);
    }
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint32_t ow[4] = {s.x[g].x, s.x[g].y, s.x[g].z, s.x[g].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float lo, hi;
        if (p.bf16) {
          lo = __uint_as_float(ow[i] << 16);
          hi = __uint_as_float(ow[i] & 0xffff0000u);
        } else {
          const __half2 hh = *reinterpret_cast<const __half2*>(&ow[i]);
          lo = __low2float(hh);
          hi = __high2float(hh);
        }
        v[g * 8 + 2 * i] += p.beta * lo;
        v[g * 8 + 2 * i + 1] += p.beta * hi;
      }
    }
  }
}
__device__ __forceinline__ uint32_t pack_out(bool bf16, float lo, float hi) {
  return bf16 ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi);
}

template <int TN>
__global__ void __launch_bounds__(192, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_y,
            const __grid_constant__ CUtensorMap tm_d, const GemmParams p) {
  using C = GemmCfg<TN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t sX = smem_base;
  const uint32_t sY = smem_base + C::NSTAGE * C::XB;
  const uint32_t sStage = sY + C::NSTAGE * C::YB;             // [2] output staging tiles
  const uint32_t sBar = sStage + 2 * C::STAGEB;
  const uint32_t bar_full = sBar;                            // [NSTAGE] leader: both CTAs' loads of a stage landed
  const uint32_t bar_empty = sBar + 8 * C::NSTAGE;           // [NSTAGE] each CTA: its stage was consumed
  const uint32_t bar_acc_full = bar_empty + 8 * C::NSTAGE;   // [2] each CTA: accumulator complete
  const uint32_t bar_acc_empty = bar_acc_full + 16;          // [2] leader: both epilogues have read it
  const uint32_t bar_staged = bar_acc_empty + 16;            // [2] a staging tile is complete (4 epilogue warps)
  const uint32_t bar_stage_free = bar_staged + 16;           // [2] the TMA store has read a staging tile
  uint8_t* gBar = smem_gen + (sBar - smem_base);
  const uint32_t off_misc = 8 * (2 * C::NSTAGE + 8);
  volatile uint32_t* s_tmem_base = reinterpret_cast<volatile uint32_t*>(gBar + off_misc);
  volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(gBar + off_misc + 4);
  const AbortCtx actx{s_abort, p.status};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t crank = cluster_ctarank(), rank = crank & 1u;   // rank within the pair; even = the pair's leader
  const int part = (int)(crank >> 1);                            // which part of the reduction (0 without a split)
  const int pair_id = (int)(blockIdx.x >> 1) / p.splits, n_pairs = (int)(gridDim.x >> 1) / p.splits;   // tiles in flight
  const int total_tiles = p.tiles_r * p.tiles_c * p.L;
  const int bk = p.tf32 ? C::BK / 2 : C::BK;   // elements per 128-byte row of a k-block
  const int nks_all = (p.K + bk * C::KSUB - 1) / (bk * C::KSUB);
  const int ks0 = nks_all * part / p.splits, nks = nks_all * (part + 1) / p.splits - ks0;   // this pair's stages of k-blocks

  cluster_arrive_started();
  if (tid == 0) {
    for (int i = 0; i < C::NSTAGE; ++i) { mbar_init(bar_full + 8 * i, 2); mbar_init(bar_empty + 8 * i, 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar_acc_full + 8 * i, 1); mbar_init(bar_acc_empty + 8 * i, 256); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar_staged + 8 * i, 4); mbar_init(bar_stage_free + 8 * i, 1); }
    *s_abort = 0u;
    fence_barrier_init();
  }
  __syncwarp();
  cluster_wait_started();
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(s_tmem_base)), 2 * TN);
    tmem_relinquish_pair();
    grid_dependency_launch();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tm_x); tma_prefetch_desc(&tm_y); tma_prefetch_desc(&tm_d); }
  grid_dependency_wait();
  tc_fence_before_sync();
  // One decision for the cluster: all CTAs skip or all run.  Its cluster barrier also says that the peer's barriers
  // exist before anything is signalled on them.
  const bool skip = cluster_should_skip(p.status, 2 * p.splits);
  tc_fence_after_sync();
  const uint32_t tmem_base = *s_tmem_base;
  if (skip) {
    if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * TN);
    return;
  }

  if (warp == 0) {
    if (lane == 0) {
      int idx = 0, local = 0;
      bool ok = true;
      for (int tile = pair_id; tile < total_tiles && ok; tile += n_pairs, ++local) {
        int tr, tc, b;
        tile_coords(tile, p.tiles_r, p.tiles_c, tr, tc, b);
        // Every other tile of a pair walks the reduction backwards: its first k-blocks are the ones the tile before
        // it (same row panels, as a rule) touched last, which are the ones still in L2.  The sum does not care.
        for (int i = 0; i < nks; ++i, ++idx) {
          const int ks = ks0 + ((local & 1) ? nks - 1 - i : i);
          const int s = idx % C::NSTAGE;
          const uint32_t ph = (idx / C::NSTAGE) & 1;
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, actx, kErrGemmEmpty)) { ok = false; break; }
          const uint32_t leader_full = map_to_cta(bar_full + 8 * s, crank & ~1u);
          mbar_arrive_expect_tx_cluster(leader_full, C::XB + C::YB);
#pragma unroll
          for (int h = 0; h < C::KSUB; ++h) {       // a k-block behind the end of K is zero-filled
            const int k = (ks * C::KSUB + h) * bk;
            tma_load_3d_pair(sX + s * C::XB + h * C::XSUB, &tm_x, leader_full, k, tr * C::TM + (int)rank * C::BM, b);
            tma_load_3d_pair(sY + s * C::YB + h * C::YSUB, &tm_y, leader_full, k, tc * TN + (int)rank * C::BNH, b);
          }
        }
      }
    }
  } else if (warp == 1) {
    // UMMA issue: all 32 lanes of the leader's warp run the loop, one elected lane executes the instructions
    if (rank == 0) {
      const uint32_t leader = elect_one();
      const uint16_t pair_mask = (uint16_t)(3u << (crank & ~1u));
      constexpr uint32_t idesc_f16 = make_idesc(1, kFmtF16, kFmtF16, 0, 0, C::TM, TN);
      constexpr uint32_t idesc_bf16 = make_idesc(1, kFmtBF16, kFmtBF16, 0, 0, C::TM, TN);
      constexpr uint32_t idesc_tf32 = make_idesc(1, 2u, 2u, 0, 0, C::TM, TN);   // kind::tf32: format code 2
      const uint32_t idesc = p.tf32 ? idesc_tf32 : (p.bf16 ? idesc_bf16 : idesc_f16);
      int idx = 0, local = 0;
      bool ok = true;
      for (int tile = pair_id; tile < total_tiles && ok; tile += n_pairs, ++local) {
        const int buf = local & 1;
        const uint32_t acc_ph = (local >> 1) & 1;
        if (!mbar_wait_warp(bar_acc_empty + 8 * buf, acc_ph ^ 1u, actx, kErrGemmAccEmpty)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d = tmem_base + buf * TN;
        for (int ks = 0; ks < nks; ++ks, ++idx) {
          const int s = idx % C::NSTAGE;
          if (!mbar_wait_warp(bar_full + 8 * s, (idx / C::NSTAGE) & 1, actx, kErrGemmFull)) { ok = false; break; }
          tc_fence_after_sync();
#pragma unroll
          for (int h = 0; h < C::KSUB; ++h) {
            const uint64_t a0 = make_smem_desc(sX + s * C::XB + h * C::XSUB, 16, 1024, kSwizzle128B);
            const uint64_t b0 = make_smem_desc(sY + s * C::YB + h * C::YSUB, 16, 1024, kSwizzle128B);
            if (p.tf32) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)   // 32 bytes of reduction per UMMA: 8 tf32 elements
                umma_ss_pair_tf32(d, desc_advance(a0, kk * 32), desc_advance(b0, kk * 32), idesc, (ks | h | kk) != 0 ? 1u : 0u,
                                  leader);
            } else {
#pragma unroll
              for (int kk = 0; kk < C::BK / 16; ++kk)
                umma_ss_e<false, true>(d, desc_advance(a0, kk * 32), desc_advance(b0, kk * 32), idesc,
                                       (ks | h | kk) != 0 ? 1u : 0u, leader);
            }
          }
          umma_commit_pair_e(bar_empty + 8 * s, pair_mask, leader);      // the stage is free in both CTAs
        }
        if (ok) umma_commit_pair_e(bar_acc_full + 8 * buf, pair_mask, leader);
      }
    }
  } else {
    // epilogue warps 2..5; warp w may touch TMEM lanes 32*(w%4) .. +31.  A tile leaves in chunks of 128 bytes per
    // row (64 columns, 32 for fp32 output): every thread turns its row's part of the accumulator into the output
    // type and writes it into a staging tile in the 128-byte swizzled layout; when the four warps have done so, one
    // thread hands the tile to a TMA store, which clips it at the edges of D.  Two staging tiles alternate.
    const int q = warp & 3;
    const int r = q * 32 + lane;                       // row within this CTA's 128 rows
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    const int row_in_tile = (int)rank * C::BM + r;
    const uint32_t leader_acc_empty = map_to_cta(bar_acc_empty, crank & ~1u);
    const int esz = p.tf32 ? 4 : 2;
    const int ccols = 128 / esz;                       // columns per chunk
    const int nchunk = TN / ccols;
    const bool storer = (warp == 2 && lane == 0);
    if (p.direct) {          // hand-over: the units other pairs will finish, [unit][4 columns][row][16 bytes]
      if (mbar_wait_warp(bar_acc_full, 0, actx, kErrGemmAccFull)) {
        tc_fence_after_sync();
        for (int u = 0; u < C::UNITS; ++u) {
          if (u % p.splits == part) continue;
          uint32_t acc[32];
          tmem_ld_x32(tmem_base + lane_base + u * 32, acc);
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < 8; ++g)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sX + u * C::UNITB + g * 2048 + r * 16),
                         "r"(acc[4 * g]), "r"(acc[4 * g + 1]), "r"(acc[4 * g + 2]), "r"(acc[4 * g + 3]) : "memory");
        }
      }
    } else {
    int local = 0;
    uint32_t n = 0;                                    // chunks staged so far: chunk n uses staging tile n & 1
    bool ok = true;
    for (int tile = pair_id; tile < total_tiles && ok; tile += n_pairs, ++local) {
      int tr, tc, b;
      tile_coords(tile, p.tiles_r, p.tiles_c, tr, tc, b);
      const int buf = local & 1;
      const int row = tr * C::TM + row_in_tile;
      const int col0 = tc * TN;
      const size_t src_at = (size_t)b * p.d_batch + (size_t)row * p.ldd + col0;
      const bool with_src = p.beta != 0.f && row < p.R;
      SourceRow src;
      if (with_src) load_source(src, p, src_at, p.Cn - col0);     // the first 32 columns, while the tile is being computed
      ok = mbar_wait_warp(bar_acc_full + 8 * buf, (local >> 1) & 1, actx, kErrGemmAccFull);
      if (!ok) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int ch = 0; ch < nchunk; ++ch, ++n) {
        const uint32_t sb = n & 1u;
        const uint32_t stage = sStage + sb * C::STAGEB;
        if (n >= 2u) {   // the store that last used this staging tile has read it
          ok = mbar_wait_warp(bar_stage_free + 8 * sb, ((n >> 1) & 1u) ^ 1u, actx, kErrGemmStageFree);
          if (!ok) break;
        }
        const uint32_t row_addr = stage + r * 128;
#pragma unroll 1
        for (int h = 0; h < ccols / 32; ++h) {         // 32 accumulator columns at a time
          uint32_t acc[32];
          const int cbase = ch * ccols + h * 32;       // first of these columns within the tile
          tmem_ld_x32(tmem_base + lane_base + buf * TN + cbase, acc);
          tmem_wait_ld();
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = p.alpha * __uint_as_float(acc[i]);
          if (with_src) {
            const SourceRow cur = src;
            if (cbase + 32 < TN) load_source(src, p, src_at + cbase + 32, p.Cn - (col0 + cbase + 32));
            add_source(v, p, cur);
          }
          // 16-byte pieces of the row, piece index XOR (row & 7): the 128-byte swizzle the TMA store undoes
          if (p.tf32) {
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              const uint32_t piece = (uint32_t)g ^ (uint32_t)(r & 7);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + piece * 16),
                           "r"(__float_as_uint(v[g * 4])), "r"(__float_as_uint(v[g * 4 + 1])),
                           "r"(__float_as_uint(v[g * 4 + 2])), "r"(__float_as_uint(v[g * 4 + 3])) : "memory");
            }
          } else {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint32_t w0 = pack_out(p.bf16, v[g * 8], v[g * 8 + 1]), w1 = pack_out(p.bf16, v[g * 8 + 2], v[g * 8 + 3]);
              const uint32_t w2 = pack_out(p.bf16, v[g * 8 + 4], v[g * 8 + 5]), w3 = pack_out(p.bf16, v[g * 8 + 6], v[g * 8 + 7]);
              const uint32_t piece = (uint32_t)(h * 4 + g) ^ (uint32_t)(r & 7);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row_addr + piece * 16), "r"(w0), "r"(w1),
                           "r"(w2), "r"(w3) : "memory");
            }
          }
        }
        if (ch == nchunk - 1) {   // the accumulator has been read: the next tile but one may overwrite it
          tc_fence_before_sync();
          mbar_arrive_cluster(leader_acc_empty + 8 * buf);
        }
        fence_proxy_async_smem();
        mbar_arrive_warp(bar_staged + 8 * sb);
        if (storer) {
          if (!mbar_wait(bar_staged + 8 * sb, (n >> 1) & 1u, actx, kErrGemmStaged)) { ok = false; }
          else {
            tma_store_3d(&tm_d, stage, col0 + ch * ccols, tr * C::TM + (int)rank * C::BM, b);
            tma_store_commit();
            tma_store_wait_read1();            // every store but this one has read its staging tile
            if (n >= 1u) mbar_arrive(bar_stage_free + 8 * (sb ^ 1u));
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
    }
    if (storer) tma_store_wait_read0();
    }
  }

  if (p.direct) {
    __syncwarp();
    cluster_sync_all();      // every CTA's accumulator is in its shared memory
    if (warp >= 2 && !*s_abort) {
      const int q = warp & 3, r = q * 32 + lane;
      int tr, tc, b;
      tile_coords(pair_id, p.tiles_r, p.tiles_c, tr, tc, b);
      const int row = tr * C::TM + (int)rank * C::BM + r;
      for (int u = part; u < C::UNITS; u += p.splits) {
        const int col = tc * TN + u * 32;
        if (col >= p.Cn) break;
        const size_t at_row = (size_t)b * p.d_batch + (size_t)row * p.ldd + col;
        SourceRow src;
        if (p.beta != 0.f && !p.trans && row < p.R) load_source(src, p, at_row, p.Cn - col);
        uint32_t acc[32];
        tmem_ld_x32(tmem_base + ((uint32_t)(q * 32) << 16) + u * 32, acc);
        tmem_wait_ld();
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.f;
        for (int o = 0; o < p.splits; ++o) {           // in the order of the reduction
          if (o == part) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += __uint_as_float(acc[i]);
            continue;
          }
          const uint32_t at = map_to_cta(sX + u * C::UNITB + r * 16, (uint32_t)(2 * o) + rank);
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float4 x = ld_shared_cluster_f32x4(at + g * 2048);
            v[4 * g] += x.x; v[4 * g + 1] += x.y; v[4 * g + 2] += x.z; v[4 * g + 3] += x.w;
          }
        }
        if (row < p.R) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] *= p.alpha;
          if (p.trans) {       // the warp's 32 rows are neighbours in D
            const size_t at = (size_t)b * p.d_batch + (size_t)col * p.ldd + row;
            // All reads ahead of the first write, which might be to the same matrix, and ahead of any use: converted one by one
            // they waited for each other (16-bit, 64 x 3088 x 1032 with beta, 14.8 us).
            if (p.beta != 0.f) {
              uint32_t old[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                old[i] = 0u;
                if (col + i < p.Cn) {
                  const size_t e = at + (size_t)i * p.ldd;
                  old[i] = p.tf32 ? reinterpret_cast<const uint32_t*>(p.src)[e] : reinterpret_cast<const uint16_t*>(p.src)[e];
                }
              }
#pragma unroll
              for (int i = 0; i < 32; ++i)
                v[i] += p.beta * (p.tf32 ? __uint_as_float(old[i])
                                         : p.bf16 ? __uint_as_float(old[i] << 16) : __half2float(__ushort_as_half((uint16_t)old[i])));
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (col + i < p.Cn) {
                if (p.tf32) reinterpret_cast<float*>(p.d)[at + (size_t)i * p.ldd] = v[i];
                else reinterpret_cast<uint16_t*>(p.d)[at + (size_t)i * p.ldd] = (uint16_t)(pack_out(p.bf16, v[i], 0.f) & 0xffffu);
              }
            }
          } else {
            if (p.beta != 0.f) add_source(v, p, src);
            if (p.tf32) {
              float* dst = reinterpret_cast<float*>(p.d) + at_row;
#pragma unroll
              for (int g = 0; g < 8; ++g)
                if (col + g * 4 < p.Cn)
                  *reinterpret_cast<float4*>(dst + g * 4) = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            } else {
              uint16_t* dst = reinterpret_cast<uint16_t*>(p.d) + at_row;
#pragma unroll
              for (int g = 0; g < 4; ++g)
                if (col + g * 8 < p.Cn)
                  *reinterpret_cast<uint4*>(dst + g * 8) =
                      make_uint4(pack_out(p.bf16, v[g * 8], v[g * 8 + 1]), pack_out(p.bf16, v[g * 8 + 2], v[g * 8 + 3]),
                                 pack_out(p.bf16, v[g * 8 + 4], v[g * 8 + 5]), pack_out(p.bf16, v[g * 8 + 6], v[g * 8 + 7]));
            }
          }
        }
        __syncwarp();        // the next unit's tcgen05.ld takes the whole warp
      }
    }
  }

  settle_if_aborted(s_abort);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();           // no CTA leaves while its peer may still read its shared memory or signal it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 2 * TN);
  }
}

struct GemmPlan { int tn, splits, trans; };

// Clusters of 2 * splits CTAs (splits = 1..4) that can be resident at once on the current device, by the largest kernel.  A
// property of the device, so it is asked for once per device and not by every thread (a thread's first call: 44.7 -> 38.7 us).
static const int* resident_clusters() {   // [splits]
  constexpr int kDevices = 64;
  static std::mutex mu;
  static std::atomic<bool> known[kDevices];
  static int table[kDevices][5];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return nullptr;
  int* n = table[dev];
  if (known[dev].load(std::memory_order_acquire)) return n;
  std::lock_guard<std::mutex> lk(mu);
  if (known[dev].load(std::memory_order_relaxed)) return n;
  for (int s = 1; s <= 4; ++s) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)(2 * s);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * s) * 256);
    cfg.blockDim = dim3(GemmCfg<256>::NTHREADS);
    cfg.dynamicSmemBytes = GemmCfg<256>::SMEM_BYTES;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    n[s] = 0;
    if (cudaFuncSetAttribute(gemm_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmCfg<256>::SMEM_BYTES) !=
            cudaSuccess || cudaOccupancyMaxActiveClusters(&n[s], gemm_kernel<256>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      n[s] = 0;
    }
  }
  known[dev].store(true, std::memory_order_release);
  return n;
}

// Tile width, split and orientation.  With two waves of 256 x 256 tiles or more, and whenever nothing else is estimated to
// be faster, 256 without a split.  Below that SMs stand idle, and the estimate decides, in us: a fixed part (launch, first
// loads, epilogue), a time per k-block of the longest chain of tiles (a narrower tile costs less, but not in proportion; rows
// whose pitch is not a multiple of 32 bytes make TMA fetch every sector's neighbour too), the exchange of a split, and for
// exchanged operands, which pay where D has few rows, the two-byte stores of each column a CTA finishes.  Every further wave
// of tiles costs its epilogue besides its k-blocks, and with rows of less than 128 bytes the load of many short rows; without
// that a short reduction went to narrow tiles in many waves: 256 x 18944 x 8 in bf16 14.1 us against 9.8 with one wave of 256,
// x 64 8.8 / 7.2, fp32 x 520 14.7 / 13.2, fp32 256 x 30000 x 8 23.2 / 13.1.  The constants are
// fits to a sweep of 24 shapes x 2 orders x 18 plans in bf16 and fp32; the plan it chose was the fastest or within 5 % of it
// for nearly all.  us before / after, bf16: 2048 x 768 x 4096 25.4 / 16.4, 16 x 3088 x 9968 50.4 / 12.8, 1408 x 536 x 2816
// 19.3 / 11.2, 88 x 88 x 80 6.9 / 5.2.
static GemmPlan plan_gemm(int R, int Cn, int K, int L, bool fp32) {
  const int* resident = resident_clusters();
  const int pairs = resident ? resident[1] : 0;
  GemmPlan best = {256, 1, 0};
  auto tiles_of = [&](int rows, int cols, int tn) { return (long long)((rows + 255) / 256) * ((cols + tn - 1) / tn) * L; };
  if (pairs <= 0 || tiles_of(R, Cn, 256) > 2 * pairs) return best;
  const long long pitch = (long long)K * (fp32 ? 4 : 2);
  const int nkb = (int)((pitch + 127) / 128);
  const bool pitch32 = pitch % 32 == 0;
  static const float fixed[3] = {6.3f, 5.3f, 4.8f};
  static const float per_kb[2][3] = {{0.37f, 0.33f, 0.29f}, {0.30f, 0.17f, 0.15f}};
  static const float wave_fixed[2][3] = {{2.3f, 1.5f, 1.0f}, {3.7f, 2.0f, 1.2f}};     // [fp32]
  static const float wave_kb[3] = {0.31f, 0.23f, 0.23f};
  const float short_rows = pitch < 128 ? 4.f * (1.f - (float)pitch / 128.f) : 0.f;
  static const float exchange[3][5] = {{0, 0, 2.8f, 3.5f, 4.4f}, {0, 0, 1.9f, 2.4f, 3.0f}, {0, 0, 1.4f, 2.1f, 2.4f}};
  float best_t = 0.f;
  for (int trans = 0; trans < 2; ++trans)
    for (int w = 0; w < 3; ++w)
      for (int s = 1; s <= 4; ++s) {
        const int tn = 256 >> w, stages = (nkb + (w ? 1 : 0)) / (w ? 2 : 1);
        const long long tiles = trans ? tiles_of(Cn, R, tn) : tiles_of(R, Cn, tn);
        if (s > stages || ((s > 1 || trans) && tiles > resident[s])) continue;
        const long long waves = (tiles + pairs - 1) / pairs;
        const float kb = (float)((nkb + s - 1) / s);
        float t = fixed[w] + per_kb[pitch32][w] * kb + exchange[w][s];
        if (waves > 1) t += (float)(waves - 1) * (fmaxf(wave_fixed[fp32][w], short_rows) + fmaxf(per_kb[pitch32][w], wave_kb[w]) * kb);
        if (trans) t += 0.3f + 0.03f * (float)(R < tn ? R : tn) / (float)s;
        if (best_t == 0.f || t < best_t) { best_t = t; best = GemmPlan{tn, s, trans}; }
      }
  return best;
}

template <int TN>
static int launch_gemm(const CUtensorMap& tm_x, const CUtensorMap& tm_y, const CUtensorMap& tm_d, const GemmParams& p,
                       int iterations, cudaStream_t stream) {
  using C = GemmCfg<TN>;
  static thread_local int attr_dev = -1;
  static thread_local int sm_count = 0;
  int dev = 0;
  if (note_cuda(cudaGetDevice(&dev), "cudaGetDevice") != cudaSuccess) return CFK_ERR_NO_DRIVER;
  if (attr_dev != dev) {
    if (note_cuda(cudaFuncSetAttribute(gemm_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES),
                  "cudaFuncSetAttribute(gemm smem)") != cudaSuccess)
      return CFK_ERR_LAUNCH;
    if (note_cuda(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev), "sm count") != cudaSuccess)
      return CFK_ERR_LAUNCH;
    attr_dev = dev;
  }
  const long long total = (long long)p.tiles_r * p.tiles_c * p.L;
  // the pairs (one per two SMs) are persistent and walk the tiles, or there is a cluster per tile
  const long long clusters = p.direct || total < sm_count / 2 ? total : sm_count / 2;
  const dim3 grid((unsigned)(2 * p.splits * clusters));
  for (int it = 0; it < iterations; ++it)
    if (note_cuda(launch_overlapped_in(2 * p.splits, gemm_kernel<TN>, grid, dim3(C::NTHREADS), C::SMEM_BYTES, stream, tm_x, tm_y,
                                       tm_d, p), "gemm launch") != cudaSuccess)
      return CFK_ERR_LAUNCH;
  return CFK_OK;
}

}  // namespace cfk

using namespace cfk;

static int check_gemm_args(const cfk_gemm_args* a) {
  if (!a || !a->a || !a->b || !a->c) return CFK_ERR_INVALID_ARG;
  if (a->m <= 0 || a->n <= 0 || a->k <= 0 || a->l <= 0 || a->iterations < 0) return CFK_ERR_INVALID_ARG;
  if (a->dtype != CFK_FP16 && a->dtype != CFK_BF16 && a->dtype != CFK_FP32) return CFK_ERR_UNSUPPORTED;
  if ((a->m % 8) || (a->n % 8) || (a->k % 8)) return CFK_ERR_UNSUPPORTED;
  if (((uintptr_t)a->a | (uintptr_t)a->b | (uintptr_t)a->c | (uintptr_t)a->c_src) & 15u) return CFK_ERR_INVALID_ARG;
  return CFK_OK;
}

extern "C" int cfk_gemm_plan(const cfk_gemm_args* a, int plan[3]) {
  const int rc = check_gemm_args(a);
  if (rc != CFK_OK || !plan) return rc != CFK_OK ? rc : CFK_ERR_INVALID_ARG;
  const GemmPlan g = a->c_row_major ? plan_gemm(a->m, a->n, a->k, a->l, a->dtype == CFK_FP32)
                                    : plan_gemm(a->n, a->m, a->k, a->l, a->dtype == CFK_FP32);
  plan[0] = g.tn; plan[1] = g.splits; plan[2] = g.trans;
  return CFK_OK;
}

extern "C" int cfk_gemm(const cfk_gemm_args* a, cfk_stream_t stream) {
  int rc = check_gemm_args(a);
  if (rc != CFK_OK) return rc;

  int err = CFK_OK;
  int* status = device_status_block(&err);
  if (!status) return err;

  // Row-major C: X = A (rows m), Y = B (rows n).  Column-major C is the row-major n x m matrix of
  // the swapped product.
  const void* x = a->c_row_major ? a->a : a->b;
  const void* y = a->c_row_major ? a->b : a->a;
  int R = a->c_row_major ? a->m : a->n;
  int Cn = a->c_row_major ? a->n : a->m;

  const GemmPlan plan = plan_gemm(R, Cn, a->k, a->l, a->dtype == CFK_FP32);

  CUtensorMap tm_x, tm_y, tm_d;
  const uint64_t esz = (uint64_t)dtype_size(a->dtype);
  const uint32_t bk = (uint32_t)(128 / esz);                   // one 128-byte span of the reduction per stage
  auto operand = [&](CUtensorMap* tm, const void* base, int rows, int box_rows) {
    const uint64_t d[3] = {(uint64_t)a->k, (uint64_t)rows, (uint64_t)a->l};
    const uint64_t st[2] = {(uint64_t)a->k * esz, (uint64_t)a->k * esz * (uint64_t)rows};
    const uint32_t box[3] = {bk, (uint32_t)box_rows, 1};
    return encode_tiled(tm, a->dtype, 3, base, d, st, box, 128);
  };
  // per CTA: 128 rows of X, and half the columns of a tile in rows of Y; `trans` exchanges the two
  if ((rc = operand(plan.trans ? &tm_y : &tm_x, x, R, plan.trans ? plan.tn / 2 : 128))) return rc;
  if ((rc = operand(plan.trans ? &tm_x : &tm_y, y, Cn, plan.trans ? 128 : plan.tn / 2))) return rc;

  // D (row-major R x Cn per batch) for the TMA store of the epilogue: boxes of 128 rows x 128 bytes
  const uint64_t dd[3] = {(uint64_t)Cn, (uint64_t)R, (uint64_t)a->l};
  const uint64_t ds[2] = {(uint64_t)Cn * esz, (uint64_t)Cn * esz * (uint64_t)R};
  const uint32_t db[3] = {bk, 128, 1};
  if ((rc = encode_tiled(&tm_d, a->dtype, 3, a->c, dd, ds, db, 128))) return rc;

  if ((long long)((R + 255) / 256) * ((Cn + 255) / 256) * a->l > 0x7fffffffLL) return CFK_ERR_UNSUPPORTED;
  GemmParams p;
  std::memset(&p, 0, sizeof(p));
  p.ldd = Cn;
  p.d_batch = (int64_t)R * Cn;
  if (plan.trans) std::swap(R, Cn);
  p.R = R; p.Cn = Cn; p.K = a->k; p.L = a->l;
  p.trans = plan.trans;
  p.direct = plan.splits > 1 || plan.trans;
  p.d = a->c;
  p.src = a->c_src ? a->c_src : a->c;
  p.alpha = a->alpha; p.beta = a->beta;
  p.bf16 = a->dtype == CFK_BF16;
  p.tf32 = a->dtype == CFK_FP32;
  p.tiles_r = (R + 255) / 256;
  p.tiles_c = (Cn + plan.tn - 1) / plan.tn;
  p.splits = plan.splits;
  p.status = status;

  switch (plan.tn) {
    case 256: return launch_gemm<256>(tm_x, tm_y, tm_d, p, a->iterations, (cudaStream_t)stream);
    case 128: return launch_gemm<128>(tm_x, tm_y, tm_d, p, a->iterations, (cudaStream_t)stream);
    default: return launch_gemm<64>(tm_x, tm_y, tm_d, p, a->iterations, (cudaStream_t)stream);
  }
}
