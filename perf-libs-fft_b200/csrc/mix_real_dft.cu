// Mixed-radix real transforms (mix_real.cuh): R2C, C2R.
#include "mix_real.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_real_dft(int kind, const MixRealLaunch& L, cudaStream_t st) {
  if (kind == FR_R2C) return run_mix_real<FR_R2C>(L, st);
  if (kind == FR_C2R) return run_mix_real<FR_C2R>(L, st);
  return cudaErrorNotSupported;
}

}  // namespace plfft_b200
