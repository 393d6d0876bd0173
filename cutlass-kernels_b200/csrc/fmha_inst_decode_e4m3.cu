// FMHA forward of a few query rows, e4m3 inputs.
#include "fmha_launch_decode_impl.cuh"

namespace cfk {

int fmha_launch_decode_e4m3(const FmhaLaunch& L, int head_dim) {
  switch (head_dim) {
    case 64: return decode_launch<kDtE4M3, kDtE4M3, 64>(L);
    case 128: return decode_launch<kDtE4M3, kDtE4M3, 128>(L);
    case 256: return decode_launch<kDtE4M3, kDtE4M3, 256>(L);
    default: return CFK_ERR_UNSUPPORTED;
  }
}

}  // namespace cfk
