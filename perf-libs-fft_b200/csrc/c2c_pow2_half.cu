// Power-of-two C2C on binary16 data, FP32 arithmetic: the compile-time stage
// list of pow2_stages.cuh between 4-byte (re, im) loads and stores of the
// user's buffers, one launch and 8 bytes of HBM traffic per element.
//
// T = N/E threads per transform, whole warps' worth of transforms per CTA.
// Bound by latency like its FP32 sibling, at half the bytes: 108 registers at
// N=1024 leave four 128-thread CTAs to an SM, 1.7 waves of the 1024 of a
// 4096-member batch.  Figures of both sides at the dispatch in plan_mix.cpp.
#include "kernels.h"
#include "launch_pdl.cuh"
#include "pow2_stages.cuh"
#include "ptx.cuh"

#include <cuda_fp16.h>

namespace plfft_b200 {

// PAIRS: both buffers 4-byte aligned; else, on an odd multiple of two bytes,
// scalar accesses
template <int N, int E, int DIR, bool PAIRS>
__global__ void __launch_bounds__(pow2_max_threads<E>(), pow2_min_blocks<E>())
    c2c_pow2_half_kernel(const Pow2HalfLaunch L) {
  griddep_wait();  // launched programmatically (launch_pdl.cuh)
  griddep_launch_dependents();
  using P = P2<N, E>;
  constexpr int T = P::T;
  constexpr int PITCH = (spad_len_c(N) + 1) & ~1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int grp = threadIdx.x / T, t = threadIdx.x - grp * T;
  const int64_t b = int64_t(blockIdx.x) * L.g + grp;
  const bool live = b < L.howmany;
  float2* buf = reinterpret_cast<float2*>(smraw) + grp * PITCH;
  auto sync = [&]() {
    if constexpr (T <= 32)
      __syncwarp();
    else
      __syncthreads();
  };
  const __half2* src = static_cast<const __half2*>(L.in) + (live ? b * L.idist : 0);
  __half2 h[E];
  if constexpr (PAIRS) {
#pragma unroll
    for (int q = 0; q < E; ++q) h[q] = live ? src[t + T * q] : __half2half2(__ushort_as_half(0));
  } else {
    const __half* s = reinterpret_cast<const __half*>(src);
#pragma unroll
    for (int q = 0; q < E; ++q)
      h[q] = live ? __halves2half2(s[2 * (t + T * q)], s[2 * (t + T * q) + 1]) : __half2half2(__ushort_as_half(0));
  }
  float2 v[E];
#pragma unroll
  for (int q = 0; q < E; ++q) v[q] = __half22float2(h[q]);
  st_bfly<T, E, P::radix(0), 1, 0, DIR>(v, t, L.tw);
  Stages<N, E, DIR, 1>::run(v, t, buf, L.tw, sync);
  if (!live) return;
  __half2* dst = static_cast<__half2*>(L.out) + b * L.odist;
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const __half2 y = __float22half2_rn(cscale(v[q], L.scale));
    if constexpr (PAIRS) {
      dst[t + T * q] = y;
    } else {
      reinterpret_cast<__half*>(dst)[2 * (t + T * q)] = __low2half(y);
      reinterpret_cast<__half*>(dst)[2 * (t + T * q) + 1] = __high2half(y);
    }
  }
}

template <int N, int E>
static cudaError_t run_half(int dir, Pow2HalfLaunch L, cudaStream_t st) {
  constexpr int T = N / E;
  L.g = T >= 128 ? 1 : 128 / T;
  const int smem = L.g * ((spad_len_c(N) + 1) & ~1) * int(sizeof(float2));
  auto k = L.pairs ? (dir < 0 ? c2c_pow2_half_kernel<N, E, -1, true> : c2c_pow2_half_kernel<N, E, 1, true>)
                   : (dir < 0 ? c2c_pow2_half_kernel<N, E, -1, false> : c2c_pow2_half_kernel<N, E, 1, false>);
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  const int64_t grid = (L.howmany + L.g - 1) / L.g;
  return launch_pdl(k, dim3(unsigned(grid)), dim3(T * L.g), size_t(smem), st, L);
}

// Elements per thread, us at 2^24 numbers a call with 8 / 16 / 32:
//   64: 36.7 / 46.6 / 80.4     128: 36.4 / 35.2 / 47.3    256: 32.8 / 23.7 / 35.5
//   512: 36.0 / 31.9 / 26.6    1024: 48.6 / 34.5 / 27.7   2048: 64.5 / 35.3 / 38.7
//   4096: 82.5 / 43.0 / 39.5   8192: - / 71.3 / 47.5
// (2^22 numbers order them alike.)
int pow2_half_e(int64_t n) { return n == 64 ? 8 : n == 128 || n == 256 || n == 2048 ? 16 : 32; }

cudaError_t launch_c2c_pow2_half(int n, int dir, const Pow2HalfLaunch& L, cudaStream_t st) {
  switch (n) {
    case 64: return run_half<64, 8>(dir, L, st);
    case 128: return run_half<128, 16>(dir, L, st);
    case 256: return run_half<256, 16>(dir, L, st);
    case 512: return run_half<512, 32>(dir, L, st);
    case 1024: return run_half<1024, 32>(dir, L, st);
    case 2048: return run_half<2048, 16>(dir, L, st);
    case 4096: return run_half<4096, 32>(dir, L, st);
    case 8192: return run_half<8192, 32>(dir, L, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace plfft_b200
