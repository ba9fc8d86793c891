// Mixed-radix real transforms (mix_real.cuh): DCT3, DST3.
#include "mix_real.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_real_dct3(int kind, const MixRealLaunch& L, cudaStream_t st) {
  if (kind == FR_DCT3) return run_mix_real<FR_DCT3>(L, st);
  if (kind == FR_DST3) return run_mix_real<FR_DST3>(L, st);
  return cudaErrorNotSupported;
}

}  // namespace plfft_b200
