// Mixed-radix real transforms (mix_real.cuh): R2HC, HC2R, DHT.
#include "mix_real.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_real_hc(int kind, const MixRealLaunch& L, cudaStream_t st) {
  if (kind == FR_R2HC) return run_mix_real<FR_R2HC>(L, st);
  if (kind == FR_HC2R) return run_mix_real<FR_HC2R>(L, st);
  if (kind == FR_DHT) return run_mix_real<FR_DHT>(L, st);
  return cudaErrorNotSupported;
}

}  // namespace plfft_b200
