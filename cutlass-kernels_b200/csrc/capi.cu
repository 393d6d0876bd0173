// C-ABI entry points that are not a kernel family of their own: argument validation and dispatch for
// cfk_fmha_forward, fills, status handling.  Declarations: include/cfk_b200.h.
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

#include "common.cuh"
#include "element_io.cuh"
#include "fmha_launch.h"
#include "host_util.h"

namespace cfk {

// ------------------------------------------------------------------------------------------------
// error text, status block, descriptor encoding
// ------------------------------------------------------------------------------------------------
static thread_local std::string g_last_error;

cudaError_t note_cuda(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
    (void)cudaGetLastError();  // clear the sticky-less error so later calls are judged on their own
  }
  return e;
}

static std::mutex g_mu;
static int* g_status_block[64] = {nullptr};

int* device_status_block(int* err) {
  int dev = -1;
  if (note_cuda(cudaGetDevice(&dev), "cudaGetDevice") != cudaSuccess || dev < 0 || dev >= 64) {
    if (err) *err = CFK_ERR_NO_DRIVER;
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_status_block[dev]) {
    int* p = nullptr;
    if (note_cuda(cudaMalloc(&p, 256), "cudaMalloc(status block)") != cudaSuccess) {
      if (err) *err = CFK_ERR_NO_DRIVER;
      return nullptr;
    }
    if (note_cuda(cudaMemset(p, 0, 256), "cudaMemset(status block)") != cudaSuccess) {
      if (err) *err = CFK_ERR_NO_DRIVER;
      return nullptr;
    }
    g_status_block[dev] = p;
  }
  return g_status_block[dev];
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (note_cuda(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres),
                  "cudaGetDriverEntryPoint(cuTensorMapEncodeTiled)") == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

int encode_tiled(CUtensorMap* map, int dtype, int rank, const void* base, const uint64_t* dims,
                 const uint64_t* strides_bytes, const uint32_t* box, int swizzle_bytes) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return CFK_ERR_NO_DRIVER;
  CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (dtype == CFK_BF16) dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  else if (dtype == CFK_E4M3) dt = CU_TENSOR_MAP_DATA_TYPE_UINT8;
  else if (dtype == CFK_FP32) dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  cuuint64_t gd[5];
  cuuint64_t gs[4];
  cuuint32_t bx[5];
  cuuint32_t es[5];
  for (int i = 0; i < rank; ++i) { gd[i] = dims[i]; bx[i] = box[i]; es[i] = 1; }
  for (int i = 0; i + 1 < rank; ++i) gs[i] = strides_bytes[i];
  CUresult r = fn(map, dt, (cuuint32_t)rank, const_cast<void*>(base), gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                  : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    g_last_error = "cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r);
    return CFK_ERR_DESCRIPTOR;
  }
  return CFK_OK;
}

int encode_bshd(CUtensorMap* map, int dtype, const void* base, int batch, int seq, int heads, int d, int64_t sb,
                int64_t ss, int64_t sh, int box_rows, int box_spans) {
  const int esz = dtype_size(dtype);
  const int span_bytes = d * esz < 128 ? d * esz : 128;   // rows shorter than 128 bytes (e4m3, d = 64) are one 64-byte span
  const uint64_t span = (uint64_t)span_bytes / esz;       // elements per span
  const uint64_t nspan = (uint64_t)d * esz / span_bytes;
  const uint64_t dims[5] = {span, (uint64_t)seq, nspan, (uint64_t)heads, (uint64_t)batch};
  const uint64_t strides[4] = {(uint64_t)ss * esz, (uint64_t)span_bytes, (uint64_t)sh * esz, (uint64_t)sb * esz};
  const uint32_t box[5] = {(uint32_t)span, (uint32_t)box_rows, (uint32_t)(box_spans > 0 ? box_spans : (int)nspan), 1, 1};
  return encode_tiled(map, dtype, 5, base, dims, strides, box, span_bytes);
}

// ------------------------------------------------------------------------------------------------
// fills
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float unit_open(uint32_t x) { return ((float)(x >> 8) + 0.5f) * (1.0f / 16777216.0f); }

__global__ void fill_kernel(void* dst, int dtype, int64_t n, uint64_t seed, int64_t first, int kind, float scale,
                            float value) {
  grid_dependency_launch();
  grid_dependency_wait();
  const uint64_t key = mix64(seed);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float v = value;
    if (kind != 2) {
      const uint64_t r = mix64(key ^ (uint64_t)(first + i));
      const float u1 = unit_open((uint32_t)r), u2 = unit_open((uint32_t)(r >> 32));
      v = (kind == 0) ? sqrtf(-2.0f * logf(u1)) * cosf(6.28318530717958647692f * u2) : 2.0f * u1 - 1.0f;
      if (kind == 3) v = rintf(v * scale);   // integers in [-scale, scale]
    }
    store_as(dst, dtype, i, kind == 3 ? v : v * scale);
  }
}

// Tunables (process-wide).  Defaults are the measured best on B200.
// EXP_EMU -1 = by type: 1 of 4 pairs for 16-bit inputs, 2 of 4 for e4m3 (measured best on B200).
// SCHED -1 = by type (see fmha_prepare).
static const int kTunableDefault[CFK_TUNE_COUNT] = {-1, 64, 0, 0, -1};
static std::atomic<int> g_tunable[CFK_TUNE_COUNT] = {{-1}, {64}, {0}, {0}, {-1}};

// The knobs can also be set from the environment (CFK_TUNE_FMHA_EXP_EMU, CFK_TUNE_FMHA_GROUP_MB, CFK_TUNE_FMHA_KERNEL,
// CFK_TUNE_FMHA_GRID, CFK_TUNE_FMHA_SCHED), read once before the first FMHA call: the command-line drivers have no flags for them.
static void tunables_from_env() {
  static std::once_flag once;
  std::call_once(once, [] {
    static const char* const names[CFK_TUNE_COUNT] = {"CFK_TUNE_FMHA_EXP_EMU", "CFK_TUNE_FMHA_GROUP_MB",
                                                      "CFK_TUNE_FMHA_KERNEL", "CFK_TUNE_FMHA_GRID",
                                                      "CFK_TUNE_FMHA_SCHED"};
    for (int i = 0; i < CFK_TUNE_COUNT; ++i) {
      const char* v = std::getenv(names[i]);
      if (v && *v) (void)cfk_set_tunable(i, std::atoi(v));
    }
  });
}

static bool valid_dtype(int dt) { return dt >= CFK_FP16 && dt <= CFK_FP32; }

}  // namespace cfk

using namespace cfk;

extern "C" int cfk_version(void) { return 100; }

extern "C" int cfk_set_tunable(int which, int value) {
  if (which < 0 || which >= CFK_TUNE_COUNT) return CFK_ERR_INVALID_ARG;
  if (value < 0) value = kTunableDefault[which];
  if (which == CFK_TUNE_FMHA_EXP_EMU && value > 3) return CFK_ERR_INVALID_ARG;
  if (which == CFK_TUNE_FMHA_GROUP_MB && (value < 1 || value > 1024)) return CFK_ERR_INVALID_ARG;
  if (which == CFK_TUNE_FMHA_KERNEL && value > 2) return CFK_ERR_INVALID_ARG;
  if (which == CFK_TUNE_FMHA_SCHED && value > 1) return CFK_ERR_INVALID_ARG;
  g_tunable[which].store(value);
  return CFK_OK;
}

extern "C" int cfk_get_tunable(int which) {
  if (which < 0 || which >= CFK_TUNE_COUNT) return -1;
  return g_tunable[which].load();
}

extern "C" const char* cfk_last_cuda_error(void) { return g_last_error.c_str(); }

extern "C" int cfk_device_status(int* code_out) {
  int err = CFK_OK;
  int* blk = device_status_block(&err);
  if (!blk) return err;
  if (note_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize") != cudaSuccess) return CFK_ERR_LAUNCH;
  int code = 0;
  if (note_cuda(cudaMemcpy(&code, blk, sizeof(int), cudaMemcpyDeviceToHost), "cudaMemcpy(status)") != cudaSuccess)
    return CFK_ERR_LAUNCH;
  if (code != 0) (void)note_cuda(cudaMemset(blk, 0, sizeof(int)), "cudaMemset(status)");
  if (code_out) *code_out = code;
  return code == 0 ? CFK_OK : CFK_ERR_DEVICE_WAIT;
}

extern "C" int cfk_fill(void* dst, int dtype, int64_t n, uint64_t seed, int64_t first_index, int kind, float scale,
                        float value, cfk_stream_t stream) {
  if (!dst || n < 0 || !valid_dtype(dtype) || kind < 0 || kind > 3) return CFK_ERR_INVALID_ARG;
  if (n == 0) return CFK_OK;
  const int threads = 256;
  const int64_t want = (n + threads - 1) / threads;
  const int blocks = (int)(want < kSMs * 16 ? want : kSMs * 16);
  return note_cuda(launch_overlapped(fill_kernel, blocks, threads, 0, (cudaStream_t)stream, dst, dtype, n, seed, first_index,
                                     kind, scale, value), "fill launch") == cudaSuccess ? CFK_OK : CFK_ERR_LAUNCH;
}

// ------------------------------------------------------------------------------------------------
// FMHA forward: validation + dispatch
// ------------------------------------------------------------------------------------------------
static bool resolve_strides(const int64_t in[3], int64_t out[3], int S, int H, int D, int esz) {
  if (in[0] == 0 && in[1] == 0 && in[2] == 0) {
    out[2] = D;
    out[1] = (int64_t)H * D;
    out[0] = (int64_t)S * H * D;
  } else {
    out[0] = in[0]; out[1] = in[1]; out[2] = in[2];
  }
  for (int i = 0; i < 3; ++i)
    if (out[i] <= 0 || (out[i] * esz) % 16 != 0) return false;
  return true;
}

// Few query rows against a long cache (fmha_decode_sm100.cuh).  It re-reads K and V per 16 query rows and its arithmetic is
// the warps' own, so it wins where the 256-row kernel has rows or SMs to spare.  us, bf16, 256-row kernel / this one:
//   up to 32 rows: d = 128, 200 heads, 8 x 1508: 43.1 / 30.1, 32 x 1532: 43.5 / 35.5; d = 64, 64 heads, 32 x 6032: 56.8 / 24.6;
//   up to 128 rows, while every group of 16 rows can have an SM: d = 128, 24 heads, 64 x 6064: 70.0 / 30.9, 8 heads,
//   128 x 1628: 22.0 / 11.4; beyond that it loses: 64 heads, 64 x 1564: 24.1 / 23.5, 200 heads, 64 x 364: 22.4 / 27.3; short
//   caches of so many rows are launch-bound either way;
//   d = 256, where the other kernel already has one 128-row tile per CTA and a tile here fills an SM: four CTAs or more per
//   group, 24 heads, 8 x 6008: 62.6 / 29.6; with fewer it is even: 64 heads, 16 x 1516: 23.4 / 25.2;
//   17 to 32 rows, two groups per head, d = 128 and 16-bit V: not where the groups run over what is resident at once (444) into
//   as many waves as the 256-row kernel has of its one CTA per head, that is with 223 to 296 heads: 256 heads, 32 x 2048:
//   54 / 66, 32 x 8192: 212 / 257; 222 and 297 heads 53 / 44 and 76 / 70.  Not so with the two-term P of bf16, which costs the
//   256-row kernel more (256 heads, 32 x 800: 38 / 36), and with e4m3 V (256 heads, 32 x 4096: 84 / 79).
static bool decode_is_faster(const cfk_fmha_args* a) {
  const int sq = a->seqlen_q, skv = a->seqlen_kv;
  const long long bh = (long long)a->batch * a->heads, groups = bh * ((sq + 15) / 16);
  if (groups > 0x7fffffffLL / 8) return false;
  if (a->head_dim == 256) return sq <= 128 && skv >= 1024 && 4 * groups <= kSMs;
  if (sq > 32) return sq <= 128 && skv >= 1024 && groups <= kSMs;
  const bool v16 = a->dtype != CFK_E4M3 || a->v_fp16;
  const int first = a->causal ? skv - sq + 1 : skv;            // keys the first row sees
  const bool two_term = a->dtype == CFK_BF16 && first < (a->p_split_keys < 0 ? 1024 : a->p_split_keys);
  if (sq > 16 && a->head_dim == 128 && v16 && !two_term && bh > kSMs) {
    const int resident = kSMs * decode_ctas_per_sm(128, dtype_size(a->dtype), 2);
    return (groups + resident - 1) / resident < (bh + kSMs - 1) / kSMs;
  }
  return true;
}

// CTAs (a cluster) per group of 16 rows: as many as are resident at once, with two tiles of keys each at least; 8 is the
// portable limit.  us for 1 / 2 / 4 / 8, bf16 d = 128: 128 heads x 6001 keys 64.2 / 62.9 / 73.9 / 70.5; 32 heads x 4096
// 30.9 / 19.9 / 16.3 / 16.0; 256 heads x 1024 24.6 / 32.5 / 33.3 / 46.1; 2 heads x 65536 410 / 210 / 108 / 57.5.
static int decode_splits(long long groups, int ntiles, int resident) {
  int s = 1;
  while (s < 8 && groups * 2 * s <= resident && ntiles >= 4 * s) s *= 2;
  return s;
}

// One 128-row tile per CTA, two CTAs per SM (fmha_fwd_tile_sm100.cuh), against one 256-row block per SM
// (fmha_fwd_sm100.cuh).  Returns the number of CTAs that share a tile's keys, 0 for the 256-row kernel.
//   Fewer tiles than CTAs fit on the chip, and at least 8 key tiles (897 keys): the keys are split as far as the chip has room,
//   two key tiles per CTA at least, eight where there is room for two parts only (8 heads, 1024 x 1024 in two: 18.4 against
//   17.0).  us, bf16 d = 128 causal, 256-row kernel / whole keys / split: 8 heads, 256 x 2048 28.4 / 25.4 / 13.7 (8 parts),
//   512 x 4096 51.2 / 46.3 / 18.8 (8), 2048 x 2048 29.0 / 28.2 / 25.9 (2); 24 heads, 512 x 4096 52.1 / 51.6 / 40.9 (2).
//   Otherwise short keys, up to 12 tiles: the estimate below decides, with 6 % in favour of the 256-row kernel.  Causal,
//   300 heads, 128 x 128 18.0 / 12.3, 300 x 300 48.4 / 33.7; 100 heads, 640 x 640 34.2 / 24.4.  With longer keys the 256-row
//   kernel, which reads K and V once per 256 rows, is as fast or faster: 8 heads, 8192 x 8192 107.5 / 120.0.
// The estimate, in us: a fixed time per CTA, a time per key tile, and for causal calls the tail of the heaviest-first order;
// the constants are fits to a sweep of 24 shapes x causal or not for each type (root mean square error 6-13 %).
struct TileCost { float fixed, per_tile, tail, offset; };
static float estimate_us(const cfk_fmha_args* a, int rows, int slots, const TileCost& c) {
  const int nq = (a->seqlen_q + rows - 1) / rows, nall = (a->seqlen_kv + 127) / 128;
  const long long bh = (long long)a->batch * a->heads, units = bh * nq;
  auto tiles_of = [&](int q) {
    const int nc = (int)(((long long)q * rows + rows - 1 + a->seqlen_kv - a->seqlen_q) / 128 + 1);
    return a->causal && nc < nall ? nc : nall;
  };
  const float longest = c.fixed + c.per_tile * (float)tiles_of(nq - 1);
  if (units <= slots) return longest + c.offset;
  if (!a->causal || nq == 1) return ceilf((float)units / (float)slots - 0.02f) * longest + c.offset;
  float sum = 0.f;
  for (int q = 0; q < nq; ++q) sum += c.fixed + c.per_tile * (float)tiles_of(q);
  const float t = sum * (float)bh / (float)slots + c.tail * (c.fixed + c.per_tile * (float)tiles_of(0));
  return (t > longest ? t : longest) + c.offset;
}

// A remainder of up to 32 rows behind the last whole block takes a CTA per head, as long as any other; without a causal mask it
// can cost a wave of its own.  It then runs in the few-rows kernel, as a second launch (about 4 us, and the cache once per 16
// rows at 1.4 times the copy rate), where the estimate says that the wave it saves is worth clearly more.  us, one launch /
// two: bf16 d = 128, 12 heads, 3080 x 3080: 83.4 / 55.6, 48 heads, 777 x 1300: 44.0 / 40.2, 75 heads, 258 x 1600: 46.7 / 39.1.
// With short keys the second launch eats the gain, so it is taken from 8 key tiles (897 keys) on (100 heads, 257 x 400: 25.3 / 26.2), and causal calls, whose CTAs differ in
// length anyway, lost (48 heads, 777 x 1300: 43.0 / 46.1).
struct TilePlan { int splits, tail_rows; };   // splits 0: the 256-row kernel
static TilePlan tile_plan(const cfk_fmha_args* a) {
  const long long bh = (long long)a->batch * a->heads, units = bh * ((a->seqlen_q + 127) / 128);
  const int nall = (a->seqlen_kv + 127) / 128;
  if (nall >= 8 && 2 * units <= 2 * kSMs) {
    int s = 2;
    while (s < 8 && units * 2 * s <= 2 * kSMs && nall >= 4 * s) s *= 2;
    if (s > 2 || nall >= 16) return TilePlan{s, 0};
  }
  if (units > 0x7fffffffLL / 4) return TilePlan{0, 0};
  static const TileCost block256[2][2] = {{{4.31f, 1.33f, 0.86f, 1.45f}, {6.33f, 1.50f, 0.88f, 1.11f}},
                                          {{3.04f, 1.38f, 0.83f, 1.13f}, {4.17f, 1.37f, 0.76f, 0.64f}}};
  static const TileCost tile128[2][2] = {{{4.60f, 1.20f, 1.09f, 1.91f}, {7.11f, 1.49f, 0.99f, 1.33f}},
                                         {{3.33f, 1.20f, 0.83f, 1.86f}, {4.40f, 1.25f, 0.71f, 1.66f}}};   // [e4m3][d = 128]
  const int e = a->dtype == CFK_E4M3 && !a->v_fp16, d = a->head_dim == 128;
  TilePlan plan{0, 0};
  if (nall <= 12 && estimate_us(a, 128, 2 * kSMs, tile128[e][d]) < 0.94f * estimate_us(a, 256, kSMs, block256[e][d]))
    plan.splits = 1;
  const int rows = plan.splits ? 128 : 256, slots = plan.splits ? 2 * kSMs : kSMs, rest = a->seqlen_q % rows;
  const long long blocks = bh * (a->seqlen_q / rows);        // whole ones
  if (!a->causal && nall >= 8 && rest > 0 && rest <= 32 && a->seqlen_q > rows) {
    const long long waves = (blocks + slots - 1) / slots, waves_all = (blocks + bh + slots - 1) / slots;
    const TileCost& c = plan.splits ? tile128[e][d] : block256[e][d];
    const float wave = c.fixed + c.per_tile * (float)nall;
    const float bytes = (float)bh * (float)((rest + 15) / 16) * (float)a->seqlen_kv * (float)a->head_dim *
                        (float)(dtype_size(a->dtype) + (a->v_fp16 ? 2 : dtype_size(a->dtype)));
    if ((float)waves * wave + 4.f + 1.4f * bytes / 6.65e6f < 0.85f * (float)waves_all * wave) plan.tail_rows = rest;
  }
  return plan;
}

static int v_dtype(const cfk_fmha_args* a) { return a->v_fp16 ? CFK_FP16 : a->dtype; }   // V, and what P is rounded to
static float descale(const cfk_fmha_args* a, float x) { return a->dtype != CFK_E4M3 && x == 0.f ? 1.f : x; }

static int check_fmha_args(const cfk_fmha_args* a) {
  if (!a || !a->q || !a->k || !a->v || !a->o) return CFK_ERR_INVALID_ARG;
  if (a->batch <= 0 || a->heads <= 0 || a->seqlen_q <= 0 || a->seqlen_kv <= 0 || a->iterations < 0)
    return CFK_ERR_INVALID_ARG;
  if (a->batch > 65535 || a->heads > 65535) return CFK_ERR_INVALID_ARG;
  if (!(a->softmax_scale > 0.f) || !std::isfinite(a->softmax_scale)) return CFK_ERR_INVALID_ARG;
  if (a->dtype != CFK_FP16 && a->dtype != CFK_BF16 && a->dtype != CFK_E4M3) return CFK_ERR_INVALID_ARG;
  if (a->out_dtype != CFK_FP16 && a->out_dtype != CFK_BF16) return CFK_ERR_INVALID_ARG;
  if (a->head_dim != 64 && a->head_dim != 128 && a->head_dim != 256) return CFK_ERR_UNSUPPORTED;
  if (a->causal && a->seqlen_kv < a->seqlen_q) return CFK_ERR_UNSUPPORTED;
  if (a->p_split_keys < -1) return CFK_ERR_INVALID_ARG;
  if (a->v_fp16 && (a->dtype != CFK_E4M3 || a->head_dim == 256)) return CFK_ERR_UNSUPPORTED;
  if (!(descale(a, a->q_descale) > 0.f) || !(descale(a, a->k_descale) > 0.f) || !(descale(a, a->v_descale) > 0.f))
    return CFK_ERR_INVALID_ARG;
  return CFK_OK;
}

// Which kernel a call runs, from its sizes, types and the knobs alone.
struct FmhaChoice {
  int variant;                    // FmhaLaunch::variant
  int splits;                     // variants 3 and 4: CTAs that share a block's keys
  int tail_rows, tail_splits;     // last rows of the call that run in the few-rows kernel, and its splits
  int sched;                      // the knob; negative: by type
};
static int few_rows_splits(const cfk_fmha_args* a, int rows) {
  const int esz = dtype_size(a->dtype), vsz = dtype_size(v_dtype(a)), keys = decode_tile_keys(a->head_dim, vsz);
  return decode_splits((long long)a->batch * a->heads * ((rows + 15) / 16), (a->seqlen_kv + keys - 1) / keys,
                       kSMs * decode_ctas_per_sm(a->head_dim, esz, vsz));
}
static FmhaChoice choose_kernel(const cfk_fmha_args* a) {
  tunables_from_env();
  FmhaChoice c = {g_tunable[CFK_TUNE_FMHA_KERNEL].load(), 0, 0, 0, g_tunable[CFK_TUNE_FMHA_SCHED].load()};
  if (c.variant == 1 && (a->dtype == CFK_E4M3 || a->head_dim != 128)) c.variant = 0;
  if (a->head_dim == 256) c.variant = 0;
  if (c.variant != 0 || c.sched >= 0 || a->s_dump) return c;   // an explicit schedule asks for the kernel that has one
  if (decode_is_faster(a)) {
    c.variant = 3;
    c.splits = few_rows_splits(a, a->seqlen_q);
  } else if (a->head_dim != 256) {
    const TilePlan plan = tile_plan(a);
    if (plan.splits > 0) c.variant = 4;
    c.splits = plan.splits;
    c.tail_rows = plan.tail_rows;
    if (c.tail_rows > 0) c.tail_splits = few_rows_splits(a, c.tail_rows);
  }
  return c;
}

extern "C" int cfk_fmha_plan(const cfk_fmha_args* a, int plan[4]) {
  const int rc = check_fmha_args(a);
  if (rc != CFK_OK || !plan) return rc != CFK_OK ? rc : CFK_ERR_INVALID_ARG;
  const FmhaChoice c = choose_kernel(a);
  plan[0] = c.variant; plan[1] = c.splits; plan[2] = c.tail_rows; plan[3] = c.tail_splits;
  return CFK_OK;
}

// Argument checks, TMA descriptors, kernel parameters and kernel choice of one FMHA call: everything of the launch
// except the status pointer and the stream, which the two entry points supply (allocated block / static array).
// *p_dtype receives the type P is rounded to (and V is stored in).
int cfk::fmha_prepare(const cfk_fmha_args* a, FmhaLaunch* out, int* p_dtype) {
  int rc = check_fmha_args(a);
  if (rc != CFK_OK) return rc;
  const int vdt = v_dtype(a);
  const uintptr_t align_or = (uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->o;
  if (align_or & 15u) return CFK_ERR_INVALID_ARG;

  const int esz = dtype_size(a->dtype);
  int64_t qs[3], ks[3], vs[3], os[3];
  if (!resolve_strides(a->q_stride, qs, a->seqlen_q, a->heads, a->head_dim, esz)) return CFK_ERR_INVALID_ARG;
  if (!resolve_strides(a->k_stride, ks, a->seqlen_kv, a->heads, a->head_dim, esz)) return CFK_ERR_INVALID_ARG;
  if (!resolve_strides(a->v_stride, vs, a->seqlen_kv, a->heads, a->head_dim, dtype_size(vdt))) return CFK_ERR_INVALID_ARG;
  if (!resolve_strides(a->o_stride, os, a->seqlen_q, a->heads, a->head_dim, 2)) return CFK_ERR_INVALID_ARG;

  FmhaLaunch& L = *out;
  std::memset(&L, 0, sizeof(L));
  const FmhaChoice choice = choose_kernel(a);
  L.variant = choice.variant;
  const bool decode = L.variant == 3;
  const int q_rows = decode ? 16 : 128, kv_rows = decode ? decode_tile_keys(a->head_dim, dtype_size(vdt)) : 128;
  if ((rc = encode_bshd(&L.tm_q, a->dtype, a->q, a->batch, a->seqlen_q, a->heads, a->head_dim, qs[0], qs[1], qs[2], q_rows)))
    return rc;
  // head dimension 256: K and V tiles travel as two halves of 128 columns (two 128-byte spans) each
  const int kv_spans = a->head_dim == 256 && !decode ? esz : 0;   // 128 columns = esz spans of 128 bytes
  if ((rc = encode_bshd(&L.tm_k, a->dtype, a->k, a->batch, a->seqlen_kv, a->heads, a->head_dim, ks[0], ks[1], ks[2], kv_rows, kv_spans)))
    return rc;
  if ((rc = encode_bshd(&L.tm_v, vdt, a->v, a->batch, a->seqlen_kv, a->heads, a->head_dim, vs[0], vs[1], vs[2], kv_rows, kv_spans)))
    return rc;
  if ((rc = encode_bshd(&L.tm_o, a->out_dtype, a->o, a->batch, a->seqlen_q, a->heads, a->head_dim, os[0], os[1], os[2], 128)))
    return rc;
  L.sp.o = a->o;
  L.sp.o_b = os[0]; L.sp.o_s = os[1]; L.sp.o_h = os[2];
  L.sp.splits = choice.splits;
  L.sp.nqb = (a->seqlen_q + 15) / 16;

  if (choice.tail_rows > 0) {   // the last rows run in the few-rows kernel
    const int keys = decode_tile_keys(a->head_dim, dtype_size(vdt));
    if ((rc = encode_bshd(&L.tail_q, a->dtype, a->q, a->batch, a->seqlen_q, a->heads, a->head_dim, qs[0], qs[1], qs[2], 16)))
      return rc;
    if ((rc = encode_bshd(&L.tail_k, a->dtype, a->k, a->batch, a->seqlen_kv, a->heads, a->head_dim, ks[0], ks[1], ks[2], keys)))
      return rc;
    if ((rc = encode_bshd(&L.tail_v, vdt, a->v, a->batch, a->seqlen_kv, a->heads, a->head_dim, vs[0], vs[1], vs[2], keys)))
      return rc;
    L.tail_rows = choice.tail_rows;
    L.tail_sp = L.sp;
    L.tail_sp.nqb = (choice.tail_rows + 15) / 16;
    L.tail_sp.row_first = a->seqlen_q - choice.tail_rows;
    L.tail_sp.splits = choice.tail_splits;
  }

  L.grid_ctas = g_tunable[CFK_TUNE_FMHA_GRID].load();
  if (L.variant == 1) {   // CTA-pair kernel: each CTA loads 64 keys of a K tile and one 64-column span of a V tile
    if ((rc = encode_bshd(&L.tm_k_half, a->dtype, a->k, a->batch, a->seqlen_kv, a->heads, a->head_dim, ks[0], ks[1], ks[2], 64)))
      return rc;
    if ((rc = encode_bshd(&L.tm_v_half, a->dtype, a->v, a->batch, a->seqlen_kv, a->heads, a->head_dim, vs[0], vs[1], vs[2], 128, 1)))
      return rc;
  }

  FmhaParams& p = L.p;
  p.B = a->batch; p.H = a->heads; p.Sq = a->seqlen_q; p.Skv = a->seqlen_kv;
  p.causal = a->causal ? 1 : 0;
  p.out_bf16 = a->out_dtype == CFK_BF16;
  // one 128-row tile per CTA at head dimension 256 and in kernels 2 and 4, two side by side otherwise
  p.nqblk = (a->head_dim == 256 || L.variant == 2 || L.variant == 4) ? (a->seqlen_q + 127) / 128 : (a->seqlen_q + 255) / 256;
  if (L.tail_rows > 0) p.nqblk -= 1;
  {
    // Default by input type, the measured best: with e4m3 Q and K the first GEMM is short enough for the two query
    // tiles to take turns on one score buffer (+8-12 % on every e4m3 shape together with the share of exponentials on
    // the FMA pipe that goes with it, below); with 16-bit inputs the hand-over of
    // the buffer would set the pace (c3 1246 -> 1221 TFLOP/s).
    p.sched = choice.sched < 0 ? (a->dtype == CFK_E4M3 ? 1 : 0) : choice.sched;
  }
  p.split_keys = a->dtype == CFK_BF16 ? (a->p_split_keys < 0 ? 1024 : a->p_split_keys) : 0;
  p.scale_log2 = a->softmax_scale * 1.4426950408889634f * descale(a, a->q_descale) * descale(a, a->k_descale);
  p.out_scale = descale(a, a->v_descale);
  p.lse = a->lse; p.mi = a->mi; p.sprime = a->sprime;
  p.s_dump = a->s_dump; p.s_dump_bf16 = a->dtype == CFK_BF16;
  L.iterations = a->iterations;
  L.exp_emu = g_tunable[CFK_TUNE_FMHA_EXP_EMU].load();
  // e4m3 at d = 128 on the shared score buffer: 1 of 4 (c5 1631 against 1486 TFLOP/s with 2 of 4 and 1386 with none)
  // 16-bit at d = 256 (one softmax warpgroup, tensor-bound): none (fp16 1302 / 1266 / 1224 / 1195 for 0..3 of 4)
  if (L.exp_emu < 0) {
    if (a->dtype != CFK_E4M3) L.exp_emu = a->head_dim == 256 ? 0 : 1;
    else L.exp_emu = (a->head_dim == 128 && (L.variant == 0 || L.variant == 4) && p.sched == 1) ? 1 : 2;
  }
  {
    // Causal: CTAs differ in length, so heads are interleaved (heaviest blocks of a group of heads first);
    // the group is sized so that its K and V stay in L2.  Non-causal: one head at a time.
    const long long kv_bytes = 2LL * a->seqlen_kv * a->head_dim * esz;
    long long grp = a->causal ? ((long long)g_tunable[CFK_TUNE_FMHA_GROUP_MB].load() << 20) / kv_bytes : 1;
    const long long bh = (long long)a->batch * a->heads;
    p.group = (int)(grp < 1 ? 1 : (grp > bh ? bh : grp));
  }
  if ((long long)p.nqblk * a->heads * a->batch > 0x7fffffffLL) return CFK_ERR_UNSUPPORTED;
  *p_dtype = vdt;
  return CFK_OK;
}

extern "C" int cfk_fmha_forward(const cfk_fmha_args* a, cfk_stream_t stream) {
  FmhaLaunch L;
  int pdt = 0;
  const int rc = fmha_prepare(a, &L, &pdt);
  if (rc != CFK_OK) return rc;
  int err = CFK_OK;
  int* status = device_status_block(&err);
  if (!status) return err;
  L.p.status = status;
  L.stream = (cudaStream_t)stream;
  return fmha_dispatch(a->dtype, pdt, a->head_dim, L);
}

#ifdef CFK_FMHA_PROFILE
// Profiling builds only: copies the 64-word status block (per-role cycle counters live in words 8..)
// to the host and clears it.
extern "C" int cfk_debug_read_status_block(int* out64) {
  int err = CFK_OK;
  int* blk = device_status_block(&err);
  if (!blk) return err;
  if (note_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize") != cudaSuccess) return CFK_ERR_LAUNCH;
  if (note_cuda(cudaMemcpy(out64, blk, 256, cudaMemcpyDeviceToHost), "cudaMemcpy(status block)") != cudaSuccess)
    return CFK_ERR_LAUNCH;
  (void)note_cuda(cudaMemset(blk, 0, 256), "cudaMemset(status block)");
  return CFK_OK;
}
#endif
