// Mixed-radix tile engine (mix.cuh): binary16 sequences around FP32 arithmetic.
#include "mix.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_f16(int dir, bool pairs, const MixLaunch<float2>& L, cudaStream_t st) {
  if (!pairs) return launch_mix_f16_scalar(dir, L, st);
  return dir < 0 ? run_mix<cpair, -1, MixIoPair<__half2, -1>>(L, st)
                 : run_mix<cpair, 1, MixIoPair<__half2, 1>>(L, st);
}

}  // namespace plfft_b200
