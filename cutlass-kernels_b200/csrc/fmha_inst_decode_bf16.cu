// FMHA forward of a few query rows, bf16 inputs.
#include "fmha_launch_decode_impl.cuh"

namespace cfk {

int fmha_launch_decode_bf16(const FmhaLaunch& L, int head_dim) {
  switch (head_dim) {
    case 64: return decode_launch<kDtBF16, kDtBF16, 64>(L);
    case 128: return decode_launch<kDtBF16, kDtBF16, 128>(L);
    case 256: return decode_launch<kDtBF16, kDtBF16, 256>(L);
    default: return CFK_ERR_UNSUPPORTED;
  }
}

}  // namespace cfk
