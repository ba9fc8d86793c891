// Mixed-radix tile engine (mix.cuh): complex FP32 sequences whose four-step
// twiddle goes by member.
#include "mix.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_f32_members(int dir, const MixLaunch<float2>& L, cudaStream_t st) {
  return dir < 0 ? run_mix<cpair, -1, MixIoPair<float2, -1, true>>(L, st)
                 : run_mix<cpair, 1, MixIoPair<float2, 1, true>>(L, st);
}

}  // namespace plfft_b200
