// Launch of one instantiation of the one-tile-per-CTA FMHA kernel (included by the fmha_inst_tile_*.cu files only).
#pragma once
#include "fmha_fwd_tile_sm100.cuh"
#include "fmha_launch.h"
#include "host_util.h"

namespace cfk {

template <int DT, int PT, int HD, int EMU>
int fmha_launch_tile_e(const FmhaLaunch& L) {
  using C = FmhaTileCfg<DT, PT, HD>;
  auto kern = fmha_fwd_tile_kernel<DT, PT, HD, EMU>;
  static thread_local int attr_set_for_device = -1;
  int dev = 0;
  if (note_cuda(cudaGetDevice(&dev), "cudaGetDevice") != cudaSuccess) return CFK_ERR_NO_DRIVER;
  if (attr_set_for_device != dev) {
    if (note_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES),
                  "cudaFuncSetAttribute(fmha tile smem)") != cudaSuccess)
      return CFK_ERR_LAUNCH;
    attr_set_for_device = dev;
  }
  FmhaSplitParams sp = L.sp;
  sp.p = L.p;
  const dim3 grid((unsigned)((long long)sp.splits * L.p.nqblk * L.p.H * L.p.B), 1, 1);
  for (int it = 0; it < L.iterations; ++it)
    if (note_cuda(launch_overlapped_in(sp.splits, kern, grid, dim3(C::NTHREADS), C::SMEM_BYTES, L.stream, L.tm_q, L.tm_k, L.tm_v,
                                       L.tm_o, sp), "fmha tile launch") != cudaSuccess)
      return CFK_ERR_LAUNCH;
  return CFK_OK;
}

template <int DT, int PT, int HD>
int fmha_launch_tile_t(const FmhaLaunch& L) {
  switch (L.exp_emu) {
    case 0: return fmha_launch_tile_e<DT, PT, HD, 0>(L);
    case 1: return fmha_launch_tile_e<DT, PT, HD, 1>(L);
    case 2: return fmha_launch_tile_e<DT, PT, HD, 2>(L);
    default: return fmha_launch_tile_e<DT, PT, HD, 3>(L);
  }
}

}  // namespace cfk
