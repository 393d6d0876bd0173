// One-tile-per-CTA FMHA forward instantiation: Q and K f16, V and P f16, head dimension 128.
#include "fmha_launch_tile_impl.cuh"

namespace cfk {
int fmha_launch_tile_f16_f16_128(const FmhaLaunch& L) { return fmha_launch_tile_t<kDtF16, kDtF16, 128>(L); }
}  // namespace cfk
