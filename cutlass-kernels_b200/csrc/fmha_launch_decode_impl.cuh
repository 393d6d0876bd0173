// Launch of one instantiation of the few-rows kernel (included by the fmha_inst_decode_*.cu files only).
#pragma once
#include "fmha_decode_sm100.cuh"
#include "fmha_launch.h"
#include "host_util.h"

namespace cfk {

template <int DT, int PT, int HD>
int decode_launch(const FmhaLaunch& L) {
  using C = DecodeCfg<DT, PT, HD>;
  auto kern = fmha_decode_kernel<DT, PT, HD>;
  static thread_local int attr_set_for_device = -1;
  int dev = 0;
  if (note_cuda(cudaGetDevice(&dev), "cudaGetDevice") != cudaSuccess) return CFK_ERR_NO_DRIVER;
  if (attr_set_for_device != dev) {
    if (note_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_MAX),
                  "cudaFuncSetAttribute(fmha decode smem)") != cudaSuccess)
      return CFK_ERR_LAUNCH;
    attr_set_for_device = dev;
  }
  FmhaSplitParams dp = L.sp;
  dp.p = L.p;
  const int ntiles = (L.p.Skv + C::TN - 1) / C::TN;
  const long long ctas = (long long)dp.splits * dp.nqb * L.p.H * L.p.B;
  dp.nslot = C::slots(ctas, kSMs, (ntiles + dp.splits - 1) / dp.splits);
  const dim3 grid((unsigned)ctas, 1, 1);
  for (int it = 0; it < L.iterations; ++it)
    if (note_cuda(launch_overlapped_in(dp.splits, kern, grid, dim3(C::NTHREADS), C::smem_bytes(dp.nslot, L.p.Sq), L.stream, L.tm_q, L.tm_k,
                                       L.tm_v, dp), "fmha decode launch") != cudaSuccess)
      return CFK_ERR_LAUNCH;
  return CFK_OK;
}

}  // namespace cfk
