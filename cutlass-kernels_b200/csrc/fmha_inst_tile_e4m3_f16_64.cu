// One-tile-per-CTA FMHA forward instantiation: Q and K e4m3, V and P f16, head dimension 64.
#include "fmha_launch_tile_impl.cuh"

namespace cfk {
int fmha_launch_tile_e4m3_f16_64(const FmhaLaunch& L) { return fmha_launch_tile_t<kDtE4M3, kDtF16, 64>(L); }
}  // namespace cfk
