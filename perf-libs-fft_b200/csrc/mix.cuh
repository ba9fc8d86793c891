// Mixed-radix tile engine: one CTA transforms a tile of sequences of one
// on-chip length, stage radices from 2..16 chosen at plan time.  FP32
// sequences go two to an engine element (cpair), FP64 ones singly.
//
// The first stage reads the user's buffer straight into registers and the
// last one writes it straight from registers; the stages between exchange
// through shared memory, one exchange per pair of stages.  What bounds it is
// latency: a tile is a chain of radix stages, and only as many bytes are in
// flight as resident threads hold.  Hence the pairs (half the index work,
// twiddle loads and operand moves per number), 80 registers and one exchange
// buffer.  C2C N=1000 x 16384 (262 MB): 149 us through the tile kernel of
// c2c.cu, 78 us with single FP32 numbers at 64 registers, 74 us with pairs at
// 128 registers and two buffers, 63 us as it is (4.1 TB/s; 66.6 us with other
// inputs on each pass).  Copying the next tile ahead into shared memory cost
// more shared-memory traffic than it hid (92 us) and was not kept.
#pragma once
#include <cuda_fp16.h>

#include "codelets.cuh"
#include "kernels.h"
#include "launch_pdl.cuh"
#include "mix.h"
#include "ptx.cuh"

namespace plfft_b200 {

__device__ __forceinline__ int mix_div(int x, uint32_t mul) { return mul ? int(__umulhi(uint32_t(x), mul)) : x; }

// element conversions between the user's type and the engine's
__device__ __forceinline__ float2 mix_cvt_in(float2 v) { return v; }
__device__ __forceinline__ float2 mix_cvt_in(__half2 v) { return __half22float2(v); }

// binary16 (re, im) that may lie on an odd multiple of two bytes
struct MixHalfPair {
  __half re, im;
};
__device__ __forceinline__ float2 mix_cvt_in(MixHalfPair v) { return make_float2(__half2float(v.re), __half2float(v.im)); }
template <class U, class V>
__device__ __forceinline__ U mix_cvt_out(V v) {
  if constexpr (std::is_same<U, __half2>::value)
    return __float22half2_rn(v);
  else if constexpr (std::is_same<U, MixHalfPair>::value)
    return MixHalfPair{__float2half_rn(v.x), __float2half_rn(v.y)};
  else
    return v;
}

// FP64 sequences in global memory
template <int DIR>
struct MixIoF64 {
  const double2* in;
  double2* out;
  int64_t ics, iks, ocs, oks;
  double scale;
  MixPost<double2> post;
  uint32_t col0;

  __device__ __forceinline__ MixIoF64(const MixLaunch<double2>& L, int64_t m, int64_t col) {
    in = static_cast<const double2*>(L.in) + m * L.ia.mdist + col * L.ia.cdist;
    out = static_cast<double2*>(L.out) + m * L.oa.mdist + col * L.oa.cdist;
    ics = L.ia.cdist;
    iks = L.ia.kstride;
    ocs = L.oa.cdist;
    oks = L.oa.kstride;
    scale = L.scale;
    post = L.post;
    col0 = uint32_t(col);
  }
  template <int R>
  __device__ __forceinline__ void load(int c, int j, int nb, double2 (&x)[R]) const {
    const double2* p = in + int64_t(c) * ics + int64_t(j) * iks;
    const int64_t step = int64_t(nb) * iks;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      x[i] = *p;
      p += step;
    }
  }
  __device__ __forceinline__ double2 finish(double2 y, int c, int k) const {
    if (post.lo) {
      const uint32_t e = (col0 + uint32_t(c)) * uint32_t(k);
      const double2 w = cmul(__ldg(post.lo + (e & ((1u << post.shift) - 1u))), __ldg(post.hi + (e >> post.shift)));
      y = twmul<DIR>(y, w);
    }
    return cscale(y, scale);
  }
  template <int R>
  __device__ __forceinline__ void store(int c, int k, int kstep, double2 (&x)[R]) const {
    double2* p = out + int64_t(c) * ocs + int64_t(k) * oks;
    const int64_t step = int64_t(kstep) * oks;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      *p = finish(x[i], c, k + i * kstep);
      p += step;
    }
  }
  __device__ __forceinline__ void store1(int c, int k, double2 y) const {
    out[int64_t(c) * ocs + int64_t(k) * oks] = finish(y, c, k);
  }
};

// FP32 arithmetic on sequences of type U, two sequences (2 c and 2 c + 1) per engine element; an odd
// last sequence rides alone, its partner a copy that is not stored
template <class U, int DIR, bool BY_MEMBER = false>
struct MixIoPair {
  const U* in;
  U* out;
  int64_t ics, iks, ocs, oks;
  float scale;
  MixPost<float2> post;
  uint32_t col0;
  int count;  // sequences of this tile
  bool wide_in, wide_out;  // both numbers of a pair lie in one aligned 16-byte word

  __device__ __forceinline__ MixIoPair(const MixLaunch<float2>& L, int64_t m, int64_t col) {
    in = static_cast<const U*>(L.in) + m * L.ia.mdist + col * L.ia.cdist;
    out = static_cast<U*>(L.out) + m * L.oa.mdist + col * L.oa.cdist;
    ics = L.ia.cdist;
    iks = L.ia.kstride;
    ocs = L.oa.cdist;
    oks = L.oa.kstride;
    scale = float(L.scale);
    post = L.post;
    col0 = uint32_t(BY_MEMBER ? m : col);
    const int64_t left = L.ncols - col;
    count = left < 2 * L.d.c ? int(left) : 2 * L.d.c;
    wide_in = L.wide_in;
    wide_out = L.wide_out;
  }
  static __device__ __forceinline__ cpair join(float2 a, float2 b) {
    return cpair{make_float2(a.x, b.x), make_float2(a.y, b.y)};
  }
  template <int R>
  __device__ __forceinline__ void load(int c, int j, int nb, cpair (&x)[R]) const {
    const U* p = in + int64_t(2 * c) * ics + int64_t(j) * iks;
    const int64_t step = int64_t(nb) * iks;
    const bool both = 2 * c + 1 < count;
    if (sizeof(U) == 8 && wide_in && both) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        x[i] = cpair{make_float2(v.x, v.z), make_float2(v.y, v.w)};
        p += step;
      }
      return;
    }
    const U* q = both ? p + ics : p;
    U u[R], v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      u[i] = *p;
      v[i] = *q;
      p += step;
      q += step;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = join(mix_cvt_in(u[i]), mix_cvt_in(v[i]));
  }
  __device__ __forceinline__ float2 twiddle(uint32_t e) const {
    return cmul(__ldg(post.lo + (e & ((1u << post.shift) - 1u))), __ldg(post.hi + (e >> post.shift)));
  }
  __device__ __forceinline__ cpair finish(cpair y, int c, int k) const {
    if (post.lo) {
      const uint32_t col = BY_MEMBER ? col0 : col0 + 2u * uint32_t(c);
      const cpair w = join(twiddle(col * uint32_t(k)),
                           twiddle((BY_MEMBER ? col : col + (2 * c + 1 < count)) * uint32_t(k)));
      const float2 wi = DIR < 0 ? w.im : fneg2(w.im);
      y = cpair{__ffma2_rn(y.im, fneg2(wi), __fmul2_rn(y.re, w.re)), __ffma2_rn(y.im, w.re, __fmul2_rn(y.re, wi))};
    }
    return cscale(y, scale);
  }
  __device__ __forceinline__ void put(U* p, bool both, cpair y) const {
    if (sizeof(U) == 8 && wide_out && both) {
      *reinterpret_cast<float4*>(p) = make_float4(y.re.x, y.im.x, y.re.y, y.im.y);
      return;
    }
    *p = mix_cvt_out<U>(make_float2(y.re.x, y.im.x));
    if (both) p[ocs] = mix_cvt_out<U>(make_float2(y.re.y, y.im.y));
  }
  template <int R>
  __device__ __forceinline__ void store(int c, int k, int kstep, cpair (&x)[R]) const {
    U* p = out + int64_t(2 * c) * ocs + int64_t(k) * oks;
    const int64_t step = int64_t(kstep) * oks;
    const bool both = 2 * c + 1 < count;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      put(p, both, finish(x[i], c, k + i * kstep));
      p += step;
    }
  }
  __device__ __forceinline__ void store1(int c, int k, cpair y) const {
    put(out + int64_t(2 * c) * ocs + int64_t(k) * oks, 2 * c + 1 < count, finish(y, c, k));
  }
};

enum MixRole { MIX_FIRST = 0, MIX_MID = 1, MIX_LAST = 2 };

// What an engine element holds, and its twiddle type: one FP64 number, one
// FP32 number of each of two transforms, or (grouped kernel) one FP32 number.
template <class V>
struct MixTraits;
template <>
struct MixTraits<double2> {
  using W = double2;
  static constexpr int lanes = 1, held = kMixHeldSingle, threads = kMixThreads64;
};
template <>
struct MixTraits<cpair> {
  using W = float2;
  static constexpr int lanes = 2, held = kMixHeldPair, threads = kMixThreadsPair;
};
template <>
struct MixTraits<float2> {
  using W = float2;
  static constexpr int lanes = 1, held = kMixHeldSingle;
};

// one 16-byte shared-memory access per element of either engine type
__device__ __forceinline__ cpair mix_ld(const cpair* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return cpair{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
template <class V>
__device__ __forceinline__ V mix_ld(const V* p) { return *p; }
__device__ __forceinline__ void mix_st(cpair* p, cpair v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
template <class V>
__device__ __forceinline__ void mix_st(V* p, V v) { *p = v; }

template <class V, int R, int DIR, int ROLE, class W, class Io>
__device__ __forceinline__ void mix_stage(const MixDesc& d, const MixStage& s, const W* __restrict__ tw, const V* src,
                                          V* dst, const Io& io, int cnt) {
  const bool cf = ROLE == MIX_FIRST ? d.cf_in : (ROLE == MIX_LAST ? d.cf_out : d.cf_mid);
  constexpr int NB = mix_held(R, MixTraits<V>::held);
  const int total = s.total, nthr = blockDim.x;
  const int tid = threadIdx.x;
  for (int f0 = 0; f0 < total; f0 += NB * nthr) {
    V x[NB][R];
    bool on[NB];
    int wpos[NB];  // shared-memory position (last stage: output index) of output 0
    int wc[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int f = f0 + b * nthr + tid;
      int c, j;
      if (cf) {
        j = mix_div(f, d.mul_c);
        c = f - j * d.c;
      } else {
        c = mix_div(f, s.mul_nb);
        j = f - c * s.nb;
      }
      on[b] = f < total && c < cnt;
      int q = j, r = 0;
      if constexpr (ROLE != MIX_FIRST) {
        q = mix_div(j, s.mul_ns);
        r = j - q * s.ns;
      }
      wc[b] = c;
      wpos[b] = ROLE == MIX_LAST ? q * (s.ns * R) + r : c * d.ld + q * s.wblk + r;
      // defined on every path: left undefined in an idle thread, the values of
      // every radix stayed live across the radix switch (a kilobyte of spills)
#pragma unroll
      for (int i = 0; i < R; ++i) x[b][i] = czero<V>();
      if (on[b]) {
        if constexpr (ROLE == MIX_FIRST) {
          io.template load<R>(c, j, s.nb, x[b]);
        } else {
          const V* p = src + c * d.ld + j + s.rpad * q;
#pragma unroll
          for (int i = 0; i < R; ++i) x[b][i] = mix_ld(p + i * s.rstep);
          const W* w = tw + s.tw_off + r;
#pragma unroll
          for (int i = 1; i < R; ++i) x[b][i] = twmul<DIR>(x[b][i], __ldg(w + (i - 1) * s.ns));
        }
      }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) dft<R, DIR>(x[b]);
    if constexpr (ROLE == MIX_MID) {
      if (d.inplace) __syncthreads();  // every read of the one buffer precedes its first write
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (!on[b]) continue;
      if constexpr (ROLE == MIX_LAST) {
        io.template store<R>(wc[b], wpos[b], s.ns, x[b]);
      } else {
        V* p = dst + wpos[b];
#pragma unroll
        for (int i = 0; i < R; ++i) mix_st(p + i * (ROLE == MIX_FIRST ? 1 : s.ns), x[b][i]);
      }
    }
  }
}

#define PLFFT_B200_MIX_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

template <class V, int DIR, int ROLE, class W, class Io>
__device__ __forceinline__ void mix_dispatch(const MixDesc& d, int si, const W* tw, const V* src, V* dst,
                                             const Io& io, int cnt) {
  const MixStage& s = d.st[si];
  switch (s.radix) {
#define PLFFT_B200_CASE(R) \
  case R:                  \
    mix_stage<V, R, DIR, ROLE>(d, s, tw, src, dst, io, cnt); \
    break;
    PLFFT_B200_MIX_RADICES(PLFFT_B200_CASE)
#undef PLFFT_B200_CASE
    default: break;
  }
}

template <class V, int DIR, class Io>
__global__ void __launch_bounds__(MixTraits<V>::threads, 1)
    mix_kernel(const __grid_constant__ MixLaunch<typename MixTraits<V>::W> L) {
  extern __shared__ __align__(16) unsigned char mix_smem[];
  griddep_wait();  // launched programmatically (launch_pdl.cuh)
  griddep_launch_dependents();
  constexpr int lanes = MixTraits<V>::lanes;
  const MixDesc& d = L.d;
  V* buf0 = reinterpret_cast<V*>(mix_smem);
  V* buf1 = d.inplace ? buf0 : buf0 + d.c * d.ld;
  const uint32_t m = blockIdx.x / L.tpm, b = blockIdx.x - m * L.tpm;
  const int64_t col = int64_t(b) * (d.c * lanes);
  const int64_t left = (L.ncols - col + lanes - 1) / lanes;
  const int cnt = left < d.c ? int(left) : d.c;
  const Io io(L, m, col);
  mix_dispatch<V, DIR, MIX_FIRST>(d, 0, L.tw, buf0, buf0, io, cnt);
  __syncthreads();
  const int ns = d.nstages;
  if (ns == 1) {
    // one stage: stored from shared memory, lanes along the dense direction
    // (C2C n=8 x 524288: 23.5 us, 37.3 with lanes along the transforms)
    const int total = d.c * d.n;
    for (int f = threadIdx.x; f < total; f += blockDim.x) {
      const int a = d.cf_out ? d.c : d.n, hi = f / a, lo = f - hi * a;
      const int k = d.cf_out ? hi : lo, c = d.cf_out ? lo : hi;
      if (c < cnt) io.store1(c, k, mix_ld(buf0 + c * d.ld + k));
    }
    return;
  }
  V* src = buf0;
  V* dst = buf1;
  for (int si = 1; si < ns - 1; ++si) {
    mix_dispatch<V, DIR, MIX_MID>(d, si, L.tw, src, dst, io, cnt);
    __syncthreads();
    V* t = src;
    src = dst;
    dst = t;
  }
  mix_dispatch<V, DIR, MIX_LAST>(d, ns - 1, L.tw, src, dst, io, cnt);
}

template <class V, int DIR, class Io>
cudaError_t run_mix(const MixLaunch<typename MixTraits<V>::W>& L, cudaStream_t st) {
  auto* k = mix_kernel<V, DIR, Io>;
  if (L.members <= 0 || L.ncols <= 0) return cudaSuccess;
  const int smem = mix_smem_bytes(L.d);
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  const int64_t grid = L.members * int64_t(L.tpm);
  if (grid > 0x7fffffff) return cudaErrorInvalidValue;
  return launch_pdl_carved(L.carveout, k, dim3(unsigned(grid)), dim3(L.d.nthr), size_t(smem), st, L);
}

}  // namespace plfft_b200
