// Scalar and packed element access by cfk_dtype, shared by the fill and the conversion kernels.  Values pass through fp32;
// results are rounded to nearest even, and saturate for e4m3.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "../../include/cfk_b200.h"

namespace cfk {

__device__ __forceinline__ void store_as(void* dst, int dtype, int64_t i, float v) {
  if (dtype == CFK_FP16) reinterpret_cast<__half*>(dst)[i] = __float2half_rn(v);
  else if (dtype == CFK_BF16) reinterpret_cast<__nv_bfloat16*>(dst)[i] = __float2bfloat16_rn(v);
  else if (dtype == CFK_E4M3)
    reinterpret_cast<uint8_t*>(dst)[i] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
  else reinterpret_cast<float*>(dst)[i] = v;
}

template <int BYTES> struct RawBytes;
template <> struct RawBytes<1> { using type = uint8_t; };
template <> struct RawBytes<2> { using type = uint16_t; };
template <> struct RawBytes<4> { using type = uint32_t; };
template <> struct RawBytes<8> { using type = uint2; };
template <> struct RawBytes<16> { using type = uint4; };

__host__ __device__ constexpr int elem_bytes(int dtype) { return dtype == CFK_E4M3 ? 1 : (dtype == CFK_FP32 ? 4 : 2); }

// V consecutive elements as one memory access of V * elem_bytes(DT) bytes
template <int DT, int V>
union ElemPack {
  typename RawBytes<V * elem_bytes(DT)>::type raw;
  float f[elem_bytes(DT) == 4 ? V : 1];
  uint16_t h[elem_bytes(DT) == 2 ? V : 1];
  uint8_t b[elem_bytes(DT) == 1 ? V : 1];
  __device__ ElemPack() {}
  __device__ __forceinline__ float get(int i) const {
    if constexpr (DT == CFK_FP32) return f[i];
    else if constexpr (DT == CFK_FP16) return __half2float(__ushort_as_half(h[i]));
    else if constexpr (DT == CFK_BF16) return __bfloat162float(__ushort_as_bfloat16(h[i]));
    else return __half2float(__half(__nv_cvt_fp8_to_halfraw(b[i], __NV_E4M3)));
  }
  __device__ __forceinline__ void set(const float (&v)[V]) {
    if constexpr (DT == CFK_FP32) {
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = v[i];
    } else if constexpr (DT == CFK_FP16) {
#pragma unroll
      for (int i = 0; i < V; ++i) h[i] = __half_as_ushort(__float2half_rn(v[i]));
    } else if constexpr (DT == CFK_BF16) {
#pragma unroll
      for (int i = 0; i < V; ++i) h[i] = __bfloat16_as_ushort(__float2bfloat16_rn(v[i]));
    } else if constexpr (V == 1) {
      b[0] = (uint8_t)__nv_cvt_float_to_fp8(v[0], __NV_SATFINITE, __NV_E4M3);
    } else {
#pragma unroll
      for (int i = 0; i < V; i += 2) {
        const __nv_fp8x2_storage_t w = __nv_cvt_float2_to_fp8x2(make_float2(v[i], v[i + 1]), __NV_SATFINITE, __NV_E4M3);
        b[i] = (uint8_t)(w & 0xffu);
        b[i + 1] = (uint8_t)(w >> 8);
      }
    }
  }
};

}  // namespace cfk
