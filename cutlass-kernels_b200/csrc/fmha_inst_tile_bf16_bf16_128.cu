// One-tile-per-CTA FMHA forward instantiation: Q and K bf16, V and P bf16, head dimension 128.
#include "fmha_launch_tile_impl.cuh"

namespace cfk {
int fmha_launch_tile_bf16_bf16_128(const FmhaLaunch& L) { return fmha_launch_tile_t<kDtBF16, kDtBF16, 128>(L); }
}  // namespace cfk
