// Mixed-radix real transforms (mix_real.cuh): DCT4, DST4.
#include "mix_real.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_real_dct4(int kind, const MixRealLaunch& L, cudaStream_t st) {
  if (kind == FR_DCT4) return run_mix_real<FR_DCT4>(L, st);
  if (kind == FR_DST4) return run_mix_real<FR_DST4>(L, st);
  return cudaErrorNotSupported;
}

}  // namespace plfft_b200
