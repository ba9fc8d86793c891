// One-kernel Rader and Bluestein transforms over lengths between the powers
// of two: the list and host-side entry points.  The kernel is in
// conv_list.cuh, instantiated per algorithm so the two compile in parallel.
#include <vector>

#include "kernels.h"

namespace plfft_b200 {

cudaError_t launch_conv_list_rader(int m, const ConvFusedLaunch& P, cudaStream_t st);
cudaError_t launch_conv_list_bluestein(int m, const ConvFusedLaunch& P, cudaStream_t st);

// (R0, A, B) in increasing order of the product.  The powers of two have their
// own kernel (conv_fused.cuh), and a length is listed only where this one beat
// it at the next power of two, 2^23 numbers a call (Bluestein, us here / there):
//   640: 98 / 100 (n=317)    768: 89 / 97 (n=383)
//   1152: 107 / 131 (n=577, Rader)   1280: 107 / 121 (n=641, Rader)   1536: 90 / 105 (n=761)
//   2304: 104 / 148 (n=1031)   2560: 96 / 125 (n=1279)   3072: 104 / 110 (n=1531)
// and for some only up to or from a batch (the rule in plan_conv.cpp).
// Not listed: 320 to 448 (132 / 125), 896 (108 / 86), 1408 and 2816 (even),
// 1664 (128 / 105), 1792, 3328, 3584 and 3840, whose larger or prime first
// radix or length eats the gain.
std::vector<int> conv_list_radices(int64_t at_least) {
  static const int lists[][3] = {
      {5, 16, 8},
      {6, 16, 8},
      {9, 16, 8},
      {10, 16, 8},
      {12, 16, 8},
      {9, 16, 16},
      {10, 16, 16},
      {12, 16, 16}};
  for (const auto& l : lists)
    if (int64_t(l[0]) * l[1] * l[2] >= at_least) return {l[0], l[1], l[2]};
  return {};
}

cudaError_t launch_conv_list(int m, bool rader, const ConvFusedLaunch& P, cudaStream_t st) {
  if (P.howmany <= 0) return cudaSuccess;
  return rader ? launch_conv_list_rader(m, P, st) : launch_conv_list_bluestein(m, P, st);
}

}  // namespace plfft_b200
