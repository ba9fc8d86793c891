// Mixed-radix real transforms: host-side entry points.  The kernel is in
// mix_real.cuh, the kinds in translation units compiled in parallel.
#include "kernels.h"
#include "mix.h"

namespace plfft_b200 {

cudaError_t launch_mix_real_dft(int kind, const MixRealLaunch& L, cudaStream_t st);
cudaError_t launch_mix_real_hc(int kind, const MixRealLaunch& L, cudaStream_t st);
cudaError_t launch_mix_real_dct2(int kind, const MixRealLaunch& L, cudaStream_t st);
cudaError_t launch_mix_real_dct3(int kind, const MixRealLaunch& L, cudaStream_t st);
cudaError_t launch_mix_real_dct4(int kind, const MixRealLaunch& L, cudaStream_t st);

bool mix_real_last_staged(int kind) { return kind != FR_C2R && kind != FR_HC2R; }

cudaError_t launch_mix_real(int kind, const MixRealLaunch& L, cudaStream_t st) {
  for (auto f : {launch_mix_real_dft, launch_mix_real_hc, launch_mix_real_dct2, launch_mix_real_dct3,
                 launch_mix_real_dct4}) {
    const cudaError_t e = f(kind, L, st);
    if (e != cudaErrorNotSupported) return e;
  }
  return cudaErrorInvalidValue;
}

}  // namespace plfft_b200
