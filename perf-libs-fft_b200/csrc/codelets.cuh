// Radix-R DFT codelets for FP32 complex data held in registers.
//
// These replace the base "codelet" kernels of the reference
// (src/providers/jit/wfta_nfact.cpp:22-171 generates the radix-2..20 DAGs
// that the AArch64 kernels evaluate; src/kernel_function_pointers.hpp:12-40
// gives their call signatures).  On the GPU a codelet is an inline device
// function over an array of R complex registers; the surrounding Stockham
// engine (stockham.cuh) supplies the data movement that the reference's
// howmany/stride loops did.
//
// Direction convention: DIR = -1 forward (exp(-2 pi i jk/R)), +1 backward.
// Constants are evaluated at compile time in double precision
// (constexpr Taylor series, own implementation) and rounded once to float.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>
#include <utility>

namespace plfft_b200 {

// ---------------------------------------------------------------------------
// complex helpers
// ---------------------------------------------------------------------------
// Complex arithmetic on float2.  sm_100 executes two FP32 lanes per
// instruction (FADD2/FMUL2/FFMA2), so re and im share one instruction.
// a - b is formed as fma(b, -1, a): exact negation, one rounding, the same
// result as a subtraction.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
// a * b = (a.x b.x - a.y b.y, a.x b.y + a.y b.x)
//       = a.x * (b.x, b.y) + a.y * (-b.y, b.x)
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  const float2 t = __fmul2_rn(make_float2(a.x, a.x), b);
  return __ffma2_rn(make_float2(a.y, a.y), make_float2(-b.y, b.x), t);
}
// a * conj(b) = a.x * (b.x, -b.y) + a.y * (b.y, b.x)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  const float2 t = __fmul2_rn(make_float2(a.x, a.x), make_float2(b.x, -b.y));
  return __ffma2_rn(make_float2(a.y, a.y), make_float2(b.y, b.x), t);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }

// Two complex FP32 numbers of two transforms side by side: (re, re) and
// (im, im) in one packed register pair each.  Complex products, rotations by
// i and sums of both transforms are then packed instructions on whole
// operands, with none of the half swaps and sign copies that a packed
// (re, im) product needs.
struct alignas(16) cpair {
  float2 re, im;
};
__device__ __forceinline__ float2 fneg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 fdup(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// The helpers below are what the codelets use, on each element type: float2
// and double2 (one complex number) and cpair (two).
template <class V>
struct ScalarOf;
template <>
struct ScalarOf<float2> {
  using type = float;
};
template <>
struct ScalarOf<double2> {
  using type = double;
};
template <>
struct ScalarOf<cpair> {
  using type = float;
};
template <class V>
using scalar_of = typename ScalarOf<V>::type;

template <class V>
__device__ __forceinline__ V czero();
template <>
__device__ __forceinline__ float2 czero<float2>() { return make_float2(0.f, 0.f); }
template <>
__device__ __forceinline__ double2 czero<double2>() { return make_double2(0.0, 0.0); }
template <>
__device__ __forceinline__ cpair czero<cpair>() { return cpair{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
__device__ __forceinline__ float2 cneg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ double2 cneg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ cpair cneg(cpair a) { return cpair{fneg2(a.re), fneg2(a.im)}; }
// s * a + b with a real s
__device__ __forceinline__ float2 cfma(float2 a, float s, float2 b) { return __ffma2_rn(a, make_float2(s, s), b); }
__device__ __forceinline__ double2 cfma(double2 a, double s, double2 b) {
  return make_double2(fma(a.x, s, b.x), fma(a.y, s, b.y));
}
__device__ __forceinline__ cpair cfma(cpair a, float s, cpair b) {
  return cpair{__ffma2_rn(a.re, fdup(s), b.re), __ffma2_rn(a.im, fdup(s), b.im)};
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ cpair cadd(cpair a, cpair b) { return cpair{__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)}; }
__device__ __forceinline__ cpair csub(cpair a, cpair b) { return cpair{fsub2(a.re, b.re), fsub2(a.im, b.im)}; }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
// both numbers of a pair times one factor w
__device__ __forceinline__ cpair cmul(cpair a, float2 w) {
  const float2 wr = fdup(w.x), wi = fdup(w.y);
  return cpair{__ffma2_rn(a.im, fneg2(wi), __fmul2_rn(a.re, wr)), __ffma2_rn(a.im, wr, __fmul2_rn(a.re, wi))};
}
__device__ __forceinline__ cpair cmulc(cpair a, float2 w) {
  const float2 wr = fdup(w.x), wi = fdup(w.y);
  return cpair{__ffma2_rn(a.im, wi, __fmul2_rn(a.re, wr)), __ffma2_rn(a.re, fneg2(wi), __fmul2_rn(a.im, wr))};
}
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ cpair cscale(cpair a, float s) {
  return cpair{__fmul2_rn(a.re, fdup(s)), __fmul2_rn(a.im, fdup(s))};
}
// times the constant (wr, wi)
__device__ __forceinline__ float2 cmulk(float2 a, float wr, float wi) { return cmul(a, make_float2(wr, wi)); }
__device__ __forceinline__ double2 cmulk(double2 a, double wr, double wi) { return cmul(a, make_double2(wr, wi)); }
__device__ __forceinline__ cpair cmulk(cpair a, float wr, float wi) { return cmul(a, make_float2(wr, wi)); }

// multiply by (s * i) where s = +1 or -1 (compile time)
template <int S>
__device__ __forceinline__ float2 cmul_i(float2 a) {
  return S > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template <int S>
__device__ __forceinline__ double2 cmul_i(double2 a) {
  return S > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}
template <int S>
__device__ __forceinline__ cpair cmul_i(cpair a) {
  return S > 0 ? cpair{fneg2(a.im), a.re} : cpair{a.im, fneg2(a.re)};
}
// (a + s i b, a - s i b)
template <int S, class V>
__device__ __forceinline__ void cadd_sub_i(V a, V b, V& sum, V& dif) {
  const V t = cmul_i<S>(b);
  sum = cadd(a, t);
  dif = csub(a, t);
}
template <int S>
__device__ __forceinline__ void cadd_sub_i(cpair a, cpair b, cpair& sum, cpair& dif) {
  const cpair p{fsub2(a.re, b.im), __fadd2_rn(a.im, b.re)}, m{__fadd2_rn(a.re, b.im), fsub2(a.im, b.re)};
  sum = S > 0 ? p : m;
  dif = S > 0 ? m : p;
}
// twiddle multiply: DIR=-1 uses the table value w, DIR=+1 uses conj(w)
template <int DIR, class V, class W>
__device__ __forceinline__ V twmul(V a, W w) {
  return DIR < 0 ? cmul(a, w) : cmulc(a, w);
}

// ---------------------------------------------------------------------------
// compile-time trigonometry (double precision)
// ---------------------------------------------------------------------------
namespace ce {
constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double sin_poly(double x) {
  // Taylor series on |x| <= pi/4, 14 terms: error far below 1 ulp of double
  double x2 = x * x, term = x, sum = x;
  for (int k = 1; k < 14; ++k) {
    term *= -x2 / double((2 * k) * (2 * k + 1));
    sum += term;
  }
  return sum;
}
constexpr double cos_poly(double x) {
  double x2 = x * x, term = 1.0, sum = 1.0;
  for (int k = 1; k < 14; ++k) {
    term *= -x2 / double((2 * k - 1) * (2 * k));
    sum += term;
  }
  return sum;
}
// cos and sin of 2*pi*k/n, exact at multiples of 1/8 turn
struct cs {
  double c, s;
};
constexpr cs unit_root(long long k, long long n) {
  k %= n;
  if (k < 0) k += n;
  // octant reduction in integer arithmetic: angle = (8k/n) * pi/4
  long long k8 = 8 * k;
  long long oct = k8 / n;          // 0..7
  long long rem = k8 - oct * n;    // angle within octant = rem/n * pi/4
  double r = double(rem) / double(n) * (kPi / 4.0);
  // reduce into [-pi/8, pi/8] style: use octant pairs
  double c0 = 0.0, s0 = 0.0;
  if (oct % 2 == 0) {
    c0 = cos_poly(r);
    s0 = sin_poly(r);
  } else {
    // angle = (oct+1)*pi/4 - (pi/4 - r)
    double r2 = kPi / 4.0 - r;
    c0 = cos_poly(r2);
    s0 = -sin_poly(r2);
    oct += 1;
  }
  // now angle = oct*pi/4 + t with cos t = c0, sin t = s0 (oct even)
  long long q = (oct / 2) % 4;
  double c = c0, s = s0;
  if (q == 1) { c = -s0; s = c0; }
  if (q == 2) { c = -c0; s = -s0; }
  if (q == 3) { c = s0; s = -c0; }
  return {c, s};
}
}  // namespace ce

// ---------------------------------------------------------------------------
// static loop helper
// ---------------------------------------------------------------------------
template <int I, int END>
struct SFor {
  template <class F>
  __device__ __forceinline__ static void run(F&& f) {
    if constexpr (I < END) {
      f(std::integral_constant<int, I>{});
      SFor<I + 1, END>::run(f);
    }
  }
};

// ---------------------------------------------------------------------------
// prime-radix codelet via symmetric pairs, R odd prime
//   X[m] = A_m + s*i*B_m,  X[R-m] = A_m - s*i*B_m
//   A_m = x0 + sum_k (x_k + x_{R-k}) cos(2 pi mk/R)
//   B_m =      sum_k (x_k - x_{R-k}) sin(2 pi mk/R)
// ---------------------------------------------------------------------------
template <int R, int DIR, class V>
__device__ __forceinline__ void dft_odd(V* v) {
  using S = scalar_of<V>;
  constexpr int H = (R - 1) / 2;
  V a[H + 1], b[H + 1];
  V x0 = v[0];
  V sum = x0;
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    a[k] = cadd(v[k], v[R - k]);
    b[k] = csub(v[k], v[R - k]);
    sum = cadd(sum, a[k]);
  }
  V out[R];
  out[0] = sum;
  SFor<1, H + 1>::run([&](auto mc) {
    constexpr int m = decltype(mc)::value;
    V A = x0, B = czero<V>();
    SFor<1, H + 1>::run([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      constexpr S c = S(ce::unit_root((m * k) % R, R).c);
      constexpr S s = S(ce::unit_root((m * k) % R, R).s);
      A = cfma(a[k], c, A);
      B = cfma(b[k], s, B);
    });
    cadd_sub_i<DIR>(A, B, out[m], out[R - m]);
  });
#pragma unroll
  for (int k = 0; k < R; ++k) v[k] = out[k];
}

template <int R, int DIR, class V>
__device__ __forceinline__ void dft(V* v);

template <int DIR, class V>
__device__ __forceinline__ void dft2(V* v) {
  V a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <int DIR, class V>
__device__ __forceinline__ void dft4(V* v) {
  V t0 = cadd(v[0], v[2]);
  V t1 = csub(v[0], v[2]);
  V t2 = cadd(v[1], v[3]);
  V t3 = csub(v[1], v[3]);
  v[0] = cadd(t0, t2);
  v[2] = csub(t0, t2);
  cadd_sub_i<DIR>(t1, t3, v[1], v[3]);
}

// composite radix R = R1 * R2 in registers:
//   n = R2*n1 + n2, k = k1 + R1*k2
//   A[n2][k1] = DFT_R1 over n1 of x[R2 n1 + n2]; A *= W_R^{n2 k1};
//   X[k1 + R1 k2] = DFT_R2 over n2 of A[n2][k1]
template <int R1, int R2, int DIR, class V>
__device__ __forceinline__ void dft_composite(V* v) {
  using S = scalar_of<V>;
  constexpr int R = R1 * R2;
  V a[R];
  SFor<0, R2>::run([&](auto n2c) {
    constexpr int n2 = decltype(n2c)::value;
    V t[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[R2 * n1 + n2];
    dft<R1, DIR>(t);
    SFor<0, R1>::run([&](auto k1c) {
      constexpr int k1 = decltype(k1c)::value;
      constexpr int e = (n2 * k1) % R;
      if constexpr (e == 0) {
        a[n2 * R1 + k1] = t[k1];
      } else if constexpr (4 * e == R) {
        a[n2 * R1 + k1] = cmul_i<DIR>(t[k1]);
      } else if constexpr (4 * e == 3 * R) {
        a[n2 * R1 + k1] = cmul_i<-DIR>(t[k1]);
      } else if constexpr (2 * e == R) {
        a[n2 * R1 + k1] = cneg(t[k1]);
      } else {
        constexpr S wr = S(ce::unit_root(e, R).c);
        constexpr S wi = S(DIR * ce::unit_root(e, R).s);
        a[n2 * R1 + k1] = cmulk(t[k1], wr, wi);
      }
    });
  });
  SFor<0, R1>::run([&](auto k1c) {
    constexpr int k1 = decltype(k1c)::value;
    V t[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) t[n2] = a[n2 * R1 + k1];
    dft<R2, DIR>(t);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = t[k2];
  });
}

template <int R, int DIR, class V>
__device__ __forceinline__ void dft(V* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    dft2<DIR>(v);
  } else if constexpr (R == 4) {
    dft4<DIR>(v);
  } else if constexpr (R == 3 || R == 5 || R == 7 || R == 11 || R == 13) {
    dft_odd<R, DIR>(v);
  } else if constexpr (R == 8) {
    dft_composite<2, 4, DIR>(v);
  } else if constexpr (R == 16) {
    dft_composite<4, 4, DIR>(v);
  } else if constexpr (R == 32) {
    dft_composite<4, 8, DIR>(v);
  } else if constexpr (R == 64) {
    dft_composite<8, 8, DIR>(v);
  } else if constexpr (R == 6) {
    dft_composite<2, 3, DIR>(v);
  } else if constexpr (R == 9) {
    dft_composite<3, 3, DIR>(v);
  } else if constexpr (R == 10) {
    dft_composite<2, 5, DIR>(v);
  } else if constexpr (R == 12) {
    dft_composite<4, 3, DIR>(v);
  } else if constexpr (R == 14) {
    dft_composite<2, 7, DIR>(v);
  } else if constexpr (R == 15) {
    dft_composite<3, 5, DIR>(v);
  } else {
    static_assert(R == 2, "unsupported radix");
  }
}

// Radices the engines can dispatch at run time.
#define PLFFT_B200_RADIX_LIST(X) X(2) X(3) X(4) X(5) X(7) X(8) X(11) X(13) X(16) X(32)

}  // namespace plfft_b200
