// Fused single-kernel real transforms for N = 2M, M a power of two: host-side
// entry points.  The kernel and its launch logic are in real_fused.cuh; the
// kinds are instantiated in three translation units compiled in parallel.
#include "kernels.h"

namespace plfft_b200 {

cudaError_t launch_real_fused_dft(int kind, int m, const RealFusedLaunch& L, cudaStream_t st);
cudaError_t launch_real_fused_dctdst23(int kind, int m, const RealFusedLaunch& L, cudaStream_t st);
cudaError_t launch_real_fused_dctdst4(int kind, int m, const RealFusedLaunch& L, cudaStream_t st);

// Elements per thread, measured on 2^25 (m = 512: 2^22) reals, us:
//   m = 2048: C2R 67.3 at 32 against 60.4 at 16, R2C 60.0 / 59.3, DCT-II
//   81.5 / 79.6, DCT-III 102 / 94; only DCT-IV is better at 32, 65.1 / 68.3;
//   m = 1024: R2C 52.2 / 59.3, DCT-II 52.5 / 77.7, DCT-IV 52.8 / 64.2, but
//   DCT-III, whose prologue holds four inputs and two factors per element,
//   125 / 99;
//   m = 512: DCT-III 17.0 at 16 against 14.7 at 8, DCT-II 11.3 / 13.2.
int real_fused_e(int kind, int m) {
  const bool iii = kind == FR_DCT3 || kind == FR_DST3, iv = kind == FR_DCT4 || kind == FR_DST4;
  if (m <= 256) return 16;
  if (m == 512) return iii ? 8 : 16;
  if (m == 1024) return iii ? 16 : 32;
  if (m == 2048) return iv ? 32 : 16;
  return m == 4096 ? 16 : 32;
}

bool real_fused_supported(int64_t m) { return m >= 64 && m <= 8192 && (m & (m - 1)) == 0; }

cudaError_t launch_real_fused(int kind, int m, const RealFusedLaunch& L, cudaStream_t st) {
  if (!real_fused_supported(m)) return cudaErrorInvalidValue;
  for (auto f : {launch_real_fused_dft, launch_real_fused_dctdst23, launch_real_fused_dctdst4}) {
    const cudaError_t e = f(kind, m, L, st);
    if (e != cudaErrorNotSupported) return e;
  }
  return cudaErrorInvalidValue;
}

}  // namespace plfft_b200
