// cfk_convert: element-wise conversion between the element types with a factor.  It replaces the host-side conversions of
// the reference's drivers (include/utils/random.hpp:20-50).
#include "common.cuh"
#include "element_io.cuh"
#include "host_util.h"

namespace cfk {

// Memory bound: every element is read and written once and nothing else is moved, so the aim is enough bytes in flight
// at whole-line accesses.  A thread moves U vectors of V elements, V chosen so that the wider of the two types travels
// as 16-byte accesses; the vectors of a block are interleaved, so that a warp's access is one contiguous piece on either
// side; all U loads are issued before the first is used.
template <int SDT, int DDT, int V, int U>
__global__ void __launch_bounds__(256) convert_kernel(const void* src, void* dst, int64_t n, float scale) {
  using S = ElemPack<SDT, V>;
  using D = ElemPack<DDT, V>;
  using SRaw = typename RawBytes<V * elem_bytes(SDT)>::type;
  using DRaw = typename RawBytes<V * elem_bytes(DDT)>::type;
  grid_dependency_launch();
  grid_dependency_wait();
  const SRaw* s = reinterpret_cast<const SRaw*>(src);
  DRaw* d = reinterpret_cast<DRaw*>(dst);
  const int64_t nvec = n / V;
  const int64_t first = (int64_t)blockIdx.x * (256 * U) + threadIdx.x;
  S in[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (first + u * 256 < nvec) in[u].raw = __ldcs(s + first + u * 256);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (first + u * 256 < nvec) {
      float v[V];
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = in[u].get(i) * scale;
      D out;
      out.set(v);
      d[first + u * 256] = out.raw;
    }
  }
  if constexpr (V > 1) {   // the elements after the last whole vector, one each for the first threads of the grid
    const int64_t i = nvec * V + (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i < n) {
      ElemPack<SDT, 1> x;
      ElemPack<DDT, 1> y;
      x.raw = reinterpret_cast<const typename RawBytes<elem_bytes(SDT)>::type*>(src)[i];
      const float v[1] = {x.get(0) * scale};
      y.set(v);
      reinterpret_cast<typename RawBytes<elem_bytes(DDT)>::type*>(dst)[i] = y.raw;
    }
  }
}

template <int SDT, int DDT>
static cudaError_t launch_convert(const void* src, void* dst, int64_t n, float scale, cudaStream_t stream) {
  constexpr int SB = elem_bytes(SDT), DB = elem_bytes(DDT);
  constexpr int V = 16 / (SB > DB ? SB : DB), U = 2, U1 = 8;
  // Vectors need both addresses to be a multiple of their own width.  Otherwise, and where the whole array is less than
  // one vector, one element per access, and more of them in flight per thread.  fp32 -> e4m3 at 67.1 M elements (335 MB): 49.7 us
  // back to back, 6.7 TB/s, against 116.9 one element at a time in a grid-stride loop.  Alone with a cold L2, by U: 1: 73.7,
  // 2: 55.3, 4: 56.2, 8: 55.3; small sizes are launch-bound.  Off by one element, by U1: 2: 136, 4: 69.2, 8: 50.1, 16: 57.2;
  // 9 M elements 19.1 / 10.3 / 7.0 / 7.9 (grid-stride loop: 125 and 11.2).
  const bool vec = n >= V && ((uintptr_t)src % (V * SB)) == 0 && ((uintptr_t)dst % (V * DB)) == 0;
  const int64_t per_block = 256 * (int64_t)(vec ? U * V : U1);
  const int64_t blocks = (n + per_block - 1) / per_block;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  auto kern = vec ? convert_kernel<SDT, DDT, V, U> : convert_kernel<SDT, DDT, 1, U1>;
  return launch_overlapped(kern, dim3((unsigned)blocks), dim3(256), 0, stream, src, dst, n, scale);
}

template <int SDT>
static cudaError_t launch_convert_to(int ddt, const void* src, void* dst, int64_t n, float scale, cudaStream_t stream) {
  switch (ddt) {
    case CFK_FP16: return launch_convert<SDT, CFK_FP16>(src, dst, n, scale, stream);
    case CFK_BF16: return launch_convert<SDT, CFK_BF16>(src, dst, n, scale, stream);
    case CFK_E4M3: return launch_convert<SDT, CFK_E4M3>(src, dst, n, scale, stream);
    default: return launch_convert<SDT, CFK_FP32>(src, dst, n, scale, stream);
  }
}

static bool valid_dtype(int dt) { return dt >= CFK_FP16 && dt <= CFK_FP32; }

}  // namespace cfk

using namespace cfk;

extern "C" int cfk_convert(const void* src, int src_dtype, void* dst, int dst_dtype, int64_t n, float scale,
                           cfk_stream_t stream) {
  if (!src || !dst || n < 0 || !valid_dtype(src_dtype) || !valid_dtype(dst_dtype)) return CFK_ERR_INVALID_ARG;
  if (n == 0) return CFK_OK;
  const cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e;
  switch (src_dtype) {
    case CFK_FP16: e = launch_convert_to<CFK_FP16>(dst_dtype, src, dst, n, scale, st); break;
    case CFK_BF16: e = launch_convert_to<CFK_BF16>(dst_dtype, src, dst, n, scale, st); break;
    case CFK_E4M3: e = launch_convert_to<CFK_E4M3>(dst_dtype, src, dst, n, scale, st); break;
    default: e = launch_convert_to<CFK_FP32>(dst_dtype, src, dst, n, scale, st); break;
  }
  return note_cuda(e, "convert launch") == cudaSuccess ? CFK_OK : CFK_ERR_LAUNCH;
}
