// Mixed-radix tile engine (mix.cuh): complex FP64 sequences.
#include "mix.cuh"

namespace plfft_b200 {

cudaError_t launch_mix_f64(int dir, const MixLaunch<double2>& L, cudaStream_t st) {
  return dir < 0 ? run_mix<double2, -1, MixIoF64<-1>>(L, st)
                 : run_mix<double2, 1, MixIoF64<1>>(L, st);
}

}  // namespace plfft_b200
