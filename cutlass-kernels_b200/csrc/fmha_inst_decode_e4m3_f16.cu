// FMHA forward of a few query rows, e4m3 Q and K, fp16 V.
#include "fmha_launch_decode_impl.cuh"

namespace cfk {

int fmha_launch_decode_e4m3_f16(const FmhaLaunch& L, int head_dim) {
  switch (head_dim) {
    case 64: return decode_launch<kDtE4M3, kDtF16, 64>(L);
    case 128: return decode_launch<kDtE4M3, kDtF16, 128>(L);
    default: return CFK_ERR_UNSUPPORTED;
  }
}

}  // namespace cfk
