// Mixed-radix tile engine (mix.cuh): binary16 sequences that are not aligned
// for 4-byte accesses.
#include "mix.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_f16_scalar(int dir, const MixLaunch<float2>& L, cudaStream_t st) {
  return dir < 0 ? run_mix<cpair, -1, MixIoPair<MixHalfPair, -1>>(L, st)
                 : run_mix<cpair, 1, MixIoPair<MixHalfPair, 1>>(L, st);
}

}  // namespace plfft_b200
