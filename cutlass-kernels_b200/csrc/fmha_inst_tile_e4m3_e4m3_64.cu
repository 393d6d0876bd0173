// One-tile-per-CTA FMHA forward instantiation: Q and K e4m3, V and P e4m3, head dimension 64.
#include "fmha_launch_tile_impl.cuh"

namespace cfk {
int fmha_launch_tile_e4m3_e4m3_64(const FmhaLaunch& L) { return fmha_launch_tile_t<kDtE4M3, kDtE4M3, 64>(L); }
}  // namespace cfk
