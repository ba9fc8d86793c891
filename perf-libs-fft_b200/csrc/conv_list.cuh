// One-kernel Rader and Bluestein transforms (the algorithm: conv_fused.cu)
// over convolution lengths between the powers of two.
//
// M = R0 A B with a small R0 and A, B in {8, 16}.  T = M / 16 threads run a
// member: radix-16 stages take one butterfly per thread and radix-8 stages
// two, so no thread idles in them.  The R0 stage is the first of the forward
// transform, where it reads the member's inputs and not the exchange buffer,
// and the last of the inverse, where it writes the outputs; in both places
// its butterflies need not be held across a barrier, so any count per thread
// will do.  The kernel is bound by the FP32 pipe, so the work saved by a
// closer M is the gain; 64 registers keep 1024 threads resident.  Bluestein
// n=1031 x 8192: 150 us at M = 4096, 104 us at M = 2304.  (Two members per
// thread in packed pairs, half the instructions at 128 registers, took 142 us:
// the pipe does the same work with fewer threads to hide it.)
#pragma once
#include "kernels.h"
#include "launch_pdl.cuh"
#include "pow2_stages.cuh"
#include "ptx.cuh"

namespace plfft_b200 {

template <int R0_, int A_, int B_>
struct ConvList {
  static constexpr int R0 = R0_, A = A_, B = B_, M = R0 * A * B, T = M / 16;
  // members per CTA: at least 96 threads
  static constexpr int G = T >= 96 ? 1 : (96 + T - 1) / T;
  static constexpr int MINB = 1024 / ((T * G + 31) / 32 * 32);
  // Exchange layouts (element k at k + P * (k / block)): the block is the
  // product of the radices done; one spare element per even block puts the
  // blocks on different banks.
  static constexpr int PF = R0 % 2 == 0 ? 1 : 0;  // forward, after R0
  static constexpr int PI = 1;                    // inverse, after A
  static constexpr int SIZE = M + (M / R0) * PF > M + (M / A) * PI ? M + (M / R0) * PF : M + (M / A) * PI;
};

// Radix-R stage of the length-M exchange buffer, held across the barrier:
// NS the product of the radices done, PIN / POUT the pads of its input (block
// NS) and output (block NS R) layouts.  put(k, value) rewrites each output.
template <int M, int T, int R, int NS, int PIN, int POUT, int DIR, class Put>
__device__ __forceinline__ void conv_stage(float2* buf, int t, const float2* __restrict__ tw, Put put) {
  constexpr int NB = M / R, H = NB / T;
  static_assert(NB % T == 0, "every thread takes H butterflies");
  float2 x[H][R];
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const int j = t + h * T, q = j / NS, r = j - q * NS;
    const float2* p = buf + j + PIN * q;
#pragma unroll
    for (int i = 0; i < R; ++i) x[h][i] = p[i * (NB + PIN * (NB / NS))];
    if constexpr (NS > 1) {
      const float2* w = tw + r;
#pragma unroll
      for (int i = 1; i < R; ++i) x[h][i] = twmul<DIR>(x[h][i], __ldg(w + (i - 1) * NS));
    }
    dft<R, DIR>(x[h]);
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const int j = t + h * T, q = j / NS, r = j - q * NS;
    float2* p = buf + q * (NS * R + POUT) + r;
#pragma unroll
    for (int i = 0; i < R; ++i) p[i * NS] = put(q * (NS * R) + r + i * NS, x[h][i]);
  }
  __syncthreads();
}

template <class L, bool RADER>
__global__ void __launch_bounds__(L::T * L::G, L::MINB) conv_list_kernel(const ConvFusedLaunch P) {
  constexpr int M = L::M, T = L::T, R0 = L::R0, A = L::A, B = L::B, NB0 = M / R0;
  extern __shared__ __align__(16) unsigned char conv_smem[];
  griddep_wait();  // launched programmatically (launch_pdl.cuh)
  griddep_launch_dependents();
  const int grp = threadIdx.x / T, t = threadIdx.x - grp * T, n = P.n;
  const int64_t b = int64_t(blockIdx.x) * L::G + grp;
  const bool live = b < P.howmany;
  // the exchange buffer and, for Rader, the member's n <= M / 2 + 1 inputs
  // (later outputs), which are permuted on chip
  constexpr int SLOT = RADER ? L::SIZE + M / 2 + 2 : L::SIZE;
  float2* buf = reinterpret_cast<float2*>(conv_smem) + grp * SLOT;
  float2* mem = buf + L::SIZE;
  const float2* in = P.in + (live ? b * P.idist : 0);
  float2 x0 = make_float2(0.f, 0.f);
  if constexpr (RADER) {
    for (int j = t; j < n; j += T) mem[j] = in[int64_t(j) * P.istride];
    __syncthreads();
    x0 = mem[0];
  }
  // forward, radix R0: element k of the zero-padded sequence
  auto elem = [&](int k) {
    if constexpr (RADER) return k < n - 1 ? mem[__ldg(P.perm_in + k)] : make_float2(0.f, 0.f);
    return k < n ? cmul(in[int64_t(k) * P.istride], __ldg(P.chirp + k)) : make_float2(0.f, 0.f);
  };
  for (int j = t; j < NB0; j += T) {
    float2 x[R0];
#pragma unroll
    for (int i = 0; i < R0; ++i) x[i] = elem(j + i * NB0);
    dft<R0, -1>(x);
    float2* p = buf + j * (R0 + L::PF);
#pragma unroll
    for (int i = 0; i < R0; ++i) p[i] = x[i];
  }
  __syncthreads();
  // tables: forward rows of A (after R0) and B (after R0 A), then the
  // inverse's rows of B (after A) and R0 (after A B)
  constexpr int TWB = (A - 1) * R0, TWIB = TWB + (B - 1) * R0 * A, TWI0 = TWIB + (B - 1) * A;
  conv_stage<M, T, A, R0, L::PF, 0, -1>(buf, t, P.tw, [](int, float2 v) { return v; });
  float2 a0 = make_float2(0.f, 0.f);  // A[0], on thread 0
  conv_stage<M, T, B, R0 * A, 0, 0, -1>(buf, t, P.tw + TWB, [&](int k, float2 v) {
    if (RADER && k == 0) a0 = v;
    return cmul(v, __ldg(P.spec + k));
  });
  // inverse: A, B, then R0 onto the outputs
  conv_stage<M, T, A, 1, 0, L::PI, 1>(buf, t, P.tw, [](int, float2 v) { return v; });
  conv_stage<M, T, B, A, L::PI, 0, 1>(buf, t, P.tw + TWIB, [](int, float2 v) { return v; });
  float2* out = P.out + b * P.odist;
  for (int j = t; j < NB0; j += T) {
    float2 x[R0];
    const float2* w = P.tw + TWI0 + j;
#pragma unroll
    for (int i = 0; i < R0; ++i) {
      x[i] = buf[j + i * NB0];
      if (i > 0) x[i] = twmul<1>(x[i], __ldg(w + (i - 1) * NB0));
    }
    dft<R0, 1>(x);
#pragma unroll
    for (int i = 0; i < R0; ++i) {
      const int k = j + i * NB0;
      if constexpr (RADER) {
        if (k < n - 1) mem[__ldg(P.perm_out + k)] = cadd(x0, x[i]);
      } else {
        if (live && k < n) out[int64_t(k) * P.ostride] = cscale(cmul(x[i], __ldg(P.chirp + k)), P.scale);
      }
    }
  }
  if constexpr (RADER) {
    if (t == 0) mem[0] = cadd(x0, a0);
    __syncthreads();
    if (live)
      for (int k = t; k < n; k += T) out[int64_t(k) * P.ostride] = cscale(mem[k], P.scale);
  }
}

template <class L, bool RADER>
cudaError_t run_conv_list(const ConvFusedLaunch& P, cudaStream_t st) {
  auto* k = conv_list_kernel<L, RADER>;
  const int smem = L::G * (RADER ? L::SIZE + L::M / 2 + 2 : L::SIZE) * int(sizeof(float2));
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(k, dim3(unsigned((P.howmany + L::G - 1) / L::G)), dim3(L::T * L::G), size_t(smem), st, P);
}

}  // namespace plfft_b200
