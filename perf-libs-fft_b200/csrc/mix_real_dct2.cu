// Mixed-radix real transforms (mix_real.cuh): DCT2, DST2.
#include "mix_real.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_real_dct2(int kind, const MixRealLaunch& L, cudaStream_t st) {
  if (kind == FR_DCT2) return run_mix_real<FR_DCT2>(L, st);
  if (kind == FR_DST2) return run_mix_real<FR_DST2>(L, st);
  return cudaErrorNotSupported;
}

}  // namespace plfft_b200
