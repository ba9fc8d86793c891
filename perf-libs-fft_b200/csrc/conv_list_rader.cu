// One-kernel Rader transforms over the listed convolution lengths (conv_list.cuh).
#include "conv_list.cuh"

namespace plfft_b200 {

cudaError_t launch_conv_list_rader(int m, const ConvFusedLaunch& P, cudaStream_t st) {
  switch (m) {
    case 640: return run_conv_list<ConvList<5, 16, 8>, true>(P, st);
    case 768: return run_conv_list<ConvList<6, 16, 8>, true>(P, st);
    case 1152: return run_conv_list<ConvList<9, 16, 8>, true>(P, st);
    case 1280: return run_conv_list<ConvList<10, 16, 8>, true>(P, st);
    case 1536: return run_conv_list<ConvList<12, 16, 8>, true>(P, st);
    case 2304: return run_conv_list<ConvList<9, 16, 16>, true>(P, st);
    case 2560: return run_conv_list<ConvList<10, 16, 16>, true>(P, st);
    case 3072: return run_conv_list<ConvList<12, 16, 16>, true>(P, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace plfft_b200
