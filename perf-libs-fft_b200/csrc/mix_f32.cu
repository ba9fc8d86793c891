// Mixed-radix tile engine (mix.cuh): complex FP32 sequences.
#include "mix.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_f32(int dir, const MixLaunch<float2>& L, cudaStream_t st) {
  return dir < 0 ? run_mix<cpair, -1, MixIoPair<float2, -1>>(L, st)
                 : run_mix<cpair, 1, MixIoPair<float2, 1>>(L, st);
}

int mix_smem_bytes(const MixDesc& d) { return d.c * d.ld * 16 * (d.inplace ? 1 : 2); }

}  // namespace plfft_b200
