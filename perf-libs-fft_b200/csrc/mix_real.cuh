// Real-data transforms of N = 2M, M any on-chip smooth length, in one pass:
// the mixed-radix tile engine (mix.cuh) with the real kinds' prologue folded
// into the first stage's loads and their epilogue into the last stage's
// stores.  The formulas are those of real_fused.cuh (which keeps the
// power-of-two M, with compile-time stage lists).
#pragma once
#include "mix.cuh"

namespace plfft_b200 {

constexpr bool mix_real_backward(int kind) {
  return kind == FR_C2R || kind == FR_HC2R || kind == FR_DCT3 || kind == FR_DST3 || kind == FR_DCT4 || kind == FR_DST4;
}
// kinds whose outputs need Z_k and Z_{M-k} together, or an output order
// other than the engine's: the last stage stays in shared memory
constexpr bool mix_real_staged(int kind) { return kind != FR_C2R && kind != FR_HC2R; }

template <int KIND>
struct MixIoReal {
  const float* in;  // first member of the tile
  float* out;
  int64_t ics, ocs;  // member distances, floats
  int m;
  float scale;
  const float2* post;  // W_N^k (DCT-IV / DST-IV: exp(i pi p / N))
  const float2* rot;   // exp(-i pi k / 2N) (DCT-IV / DST-IV: exp(i pi (4q+1) / 4N))
  int wmode, pairs_in, pairs_out;
  int count;  // members of this tile

  __device__ __forceinline__ MixIoReal(const MixRealLaunch& L, int64_t col) {
    const int64_t left = L.howmany - col;
    count = left < 2 * L.d.c ? int(left) : 2 * L.d.c;
    m = L.d.n;
    ics = L.idist * (KIND == FR_C2R ? 2 : 1);
    ocs = L.odist * (KIND == FR_R2C ? 2 : 1);
    in = static_cast<const float*>(L.in) + col * ics;
    out = static_cast<float*>(L.out) + col * ocs;
    scale = L.scale;
    post = L.post;
    rot = L.rot;
    wmode = L.wmode;
    pairs_in = L.pairs_in;
    pairs_out = L.pairs_out;
  }
  // Z'_k of a Hermitian half spectrum: (a + conj b) + i conj(w) (a - conj b)
  static __device__ __forceinline__ float2 merge(float2 xk, float2 xm, float2 w) {
    const float2 cm = make_float2(xm.x, -xm.y);
    const float2 a = cadd(xk, cm);
    const float2 d = csub(xk, cm);
    const float2 wd = cmulc(d, w);
    return cadd(a, make_float2(-wd.y, wd.x));
  }
  // element k of the complex sequence the engine transforms
  __device__ __forceinline__ float2 elem(const float* x, int k) const {
    const int n = 2 * m;
    if constexpr (KIND == FR_R2C || KIND == FR_R2HC || KIND == FR_DHT) {
      if (pairs_in) return reinterpret_cast<const float2*>(x)[k];
      return make_float2(x[2 * k], x[2 * k + 1]);
    } else if constexpr (KIND == FR_C2R) {
      const float2* X = reinterpret_cast<const float2*>(x);
      const bool k0 = k == 0;  // imaginary parts of X_0 and X_M ignored
      const float w = (wmode == 1 && !k0) ? 0.5f : 1.f;
      float2 xk = X[k], xm = X[m - k];
      xk = make_float2(xk.x * w, k0 ? 0.f : xk.y * w);
      xm = make_float2(xm.x * w, k0 ? 0.f : xm.y * w);
      return merge(xk, xm, __ldg(post + k));
    } else if constexpr (KIND == FR_HC2R) {
      const bool k0 = k == 0;
      const float2 xk = make_float2(x[k], k0 ? 0.f : x[k0 ? 0 : n - k]);
      const float2 xm = make_float2(x[m - k], k0 ? 0.f : x[k0 ? 0 : m + k]);
      return merge(xk, xm, __ldg(post + k));
    } else if constexpr (KIND == FR_DCT2 || KIND == FR_DST2) {
      // Makhoul's order v_j = x_{2j} (j < M), v_{N-1-j} = x_{2j+1}, taken in
      // pairs; DST-II: odd inputs negated
      auto v = [&](int j) {
        const float a = x[j < m ? 2 * j : 2 * (n - 1 - j) + 1];
        return (KIND == FR_DST2 && j >= m) ? -a : a;
      };
      return make_float2(v(2 * k), v(2 * k + 1));
    } else if constexpr (KIND == FR_DCT3 || KIND == FR_DST3) {
      const float w0 = wmode == 3 ? 2.f : 1.f;
      auto y = [&](int j) {  // y_N = 0
        if (j >= n) return 0.f;
        const float a = x[KIND == FR_DST3 ? n - 1 - j : j];
        return j == 0 ? w0 * a : a;
      };
      auto wk = [&](int j) { return cmulc(make_float2(y(j), -y(n - j)), __ldg(rot + j)); };
      float2 xk = wk(k), xm = wk(m - k);
      if (k == 0) xk.y = xm.y = 0.f;
      return merge(xk, xm, __ldg(post + k));
    } else {  // DCT-IV / DST-IV
      const float a = x[KIND == FR_DST4 ? n - 1 - 2 * k : 2 * k];
      const float b = x[KIND == FR_DST4 ? 2 * k : n - 1 - 2 * k];
      return cmul(make_float2(a, -b), __ldg(post + k));
    }
  }
  // members 2 c and 2 c + 1 (an odd last one with a copy of itself)
  template <int R>
  __device__ __forceinline__ void load(int c, int j, int nb, cpair (&z)[R]) const {
    const float* x0 = in + int64_t(2 * c) * ics;
    const float* x1 = 2 * c + 1 < count ? x0 + ics : x0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float2 a = elem(x0, j + i * nb), b = elem(x1, j + i * nb);
      z[i] = cpair{make_float2(a.x, b.x), make_float2(a.y, b.y)};
    }
  }
  __device__ __forceinline__ void store1(int c, int k, cpair z) const {
    z = cscale(z, scale);
    put_pair(2 * c, k, make_float2(z.re.x, z.im.x));
    if (2 * c + 1 < count) put_pair(2 * c + 1, k, make_float2(z.re.y, z.im.y));
  }
  __device__ __forceinline__ void put_pair(int b, int k, float2 z) const {
    float* y = out + int64_t(b) * ocs;
    if (pairs_out) {
      reinterpret_cast<float2*>(y)[k] = z;
    } else {
      y[2 * k] = z.x;
      y[2 * k + 1] = z.y;
    }
  }
  template <int R>
  __device__ __forceinline__ void store(int c, int k, int kstep, cpair (&z)[R]) const {
#pragma unroll
    for (int i = 0; i < R; ++i) store1(c, k + i * kstep, z[i]);
  }
  // outputs of bin k from V_k, k = 0..M
  __device__ __forceinline__ void emit(float* y, int k, float2 v) const {
    const int n = 2 * m;
    const bool inner = k > 0 && k < m;
    if constexpr (KIND == FR_R2C) {
      reinterpret_cast<float2*>(y)[k] = cscale(v, (wmode == 2 && inner) ? 2.f * scale : scale);
    } else if constexpr (KIND == FR_R2HC || KIND == FR_DHT) {
      y[k] = (KIND == FR_R2HC ? v.x : v.x - v.y) * scale;
      if (inner) y[n - k] = (KIND == FR_R2HC ? v.y : v.x + v.y) * scale;
    } else {
      const float2 c = cmul(__ldg(rot + k), v);
      const float a = 2.f * c.x * scale, b = -2.f * c.y * scale;
      if constexpr (KIND == FR_DCT2) {
        y[k] = a;
        if (inner) y[n - k] = b;
      } else {
        y[n - 1 - k] = a;
        if (inner) y[k - 1] = b;
      }
    }
  }
  static __device__ __forceinline__ float2 lane(const cpair& z, int l) {
    return l ? make_float2(z.re.y, z.im.y) : make_float2(z.re.x, z.im.x);
  }
  // epilogue of the staged kinds: Z of the tile in natural order, pitch ld
  __device__ __forceinline__ void finish(const cpair* z, int ld, int c_tile, uint32_t mul_half, uint32_t mul_m) const {
    const int n = 2 * m;
    if constexpr (KIND == FR_R2C || KIND == FR_R2HC || KIND == FR_DHT || KIND == FR_DCT2 || KIND == FR_DST2) {
      // pairs (k, M - k), k <= M / 2: V_k = e - i w o, V_{M-k} = conj(e + i w o)
      const int half = m / 2 + 1;
      for (int f = threadIdx.x; f < c_tile * half; f += blockDim.x) {
        const int c = mix_div(f, mul_half), k = f - c * half;
        const cpair pk = mix_ld(z + c * ld + k), pm = mix_ld(z + c * ld + (k ? m - k : 0));
        const float2 w = __ldg(post + k);
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          if (2 * c + l >= count) continue;
          const float2 zk = lane(pk, l), zm = lane(pm, l);
          const float2 cm = make_float2(zm.x, -zm.y);
          const float2 e = cscale(cadd(zk, cm), 0.5f);
          const float2 o = cscale(csub(zk, cm), 0.5f);
          const float2 wo = cmul(w, o);
          float* y = out + int64_t(2 * c + l) * ocs;
          emit(y, k, make_float2(e.x + wo.y, e.y - wo.x));
          if (2 * k != m) emit(y, m - k, make_float2(e.x - wo.y, -(e.y + wo.x)));
        }
      }
    } else if constexpr (KIND == FR_DCT3 || KIND == FR_DST3) {
      // u_{2j} = Re z_j, u_{2j+1} = Im z_j; x_{2j} = u_j, x_{2j+1} = u_{N-1-j}
      for (int f = threadIdx.x; f < c_tile * m; f += blockDim.x) {
        const int c = mix_div(f, mul_m), p = f - c * m, q = n - 1 - p;
        const cpair a = mix_ld(z + c * ld + (p >> 1)), b = mix_ld(z + c * ld + (q >> 1));
        const float2 ua = (p & 1) ? a.im : a.re, ub = (q & 1) ? b.im : b.re;  // of both members
        const float sb = KIND == FR_DST3 ? -scale : scale;
        if (2 * c < count) put_pair(2 * c, p, make_float2(ua.x * scale, ub.x * sb));
        if (2 * c + 1 < count) put_pair(2 * c + 1, p, make_float2(ua.y * scale, ub.y * sb));
      }
    } else {
      // S_q = rot_q C_q: y_{2q} = 2 Re S_q, y_{N-1-2q} = +-2 Im S_q, written
      // as the pairs (y_{2p}, y_{2p+1}), the second from q = M - 1 - p
      for (int f = threadIdx.x; f < c_tile * m; f += blockDim.x) {
        const int c = mix_div(f, mul_m), p = f - c * m, q = m - 1 - p;
        const cpair a = cmul(mix_ld(z + c * ld + p), __ldg(rot + p));
        const cpair b = cmul(mix_ld(z + c * ld + q), __ldg(rot + q));
        const float sa = 2.f * scale, sb = KIND == FR_DST4 ? -2.f * scale : 2.f * scale;
        if (2 * c < count) put_pair(2 * c, p, make_float2(a.re.x * sa, b.im.x * sb));
        if (2 * c + 1 < count) put_pair(2 * c + 1, p, make_float2(a.re.y * sa, b.im.y * sb));
      }
    }
  }
};

template <int KIND>
__global__ void __launch_bounds__(kMixThreadsPair, 1)
    mix_real_kernel(const __grid_constant__ MixRealLaunch L) {
  constexpr int DIR = mix_real_backward(KIND) ? 1 : -1;
  extern __shared__ __align__(16) unsigned char mix_smem[];
  griddep_wait();  // launched programmatically (launch_pdl.cuh)
  griddep_launch_dependents();
  const MixDesc& d = L.d;
  cpair* src = reinterpret_cast<cpair*>(mix_smem);
  cpair* dst = d.inplace ? src : src + d.c * d.ld;
  const MixIoReal<KIND> io(L, int64_t(blockIdx.x) * (2 * d.c));
  const int cnt = (io.count + 1) / 2;
  mix_dispatch<cpair, DIR, MIX_FIRST>(d, 0, L.tw, src, src, io, cnt);
  __syncthreads();
  const int ns = d.nstages;
  const int mid = mix_real_staged(KIND) ? ns : ns - 1;
  for (int si = 1; si < mid; ++si) {
    mix_dispatch<cpair, DIR, MIX_MID>(d, si, L.tw, src, dst, io, cnt);
    __syncthreads();
    cpair* t = src;
    src = dst;
    dst = t;
  }
  if constexpr (mix_real_staged(KIND)) {
    io.finish(src, d.ld, cnt, L.mul_half, L.mul_m);
  } else if (ns == 1) {
    for (int f = threadIdx.x; f < d.c * d.n; f += blockDim.x) {
      const int c = mix_div(f, L.mul_m), k = f - c * d.n;
      if (c < cnt) io.store1(c, k, src[c * d.ld + k]);
    }
  } else {
    mix_dispatch<cpair, DIR, MIX_LAST>(d, ns - 1, L.tw, src, dst, io, cnt);
  }
}

template <int KIND>
cudaError_t run_mix_real(const MixRealLaunch& L, cudaStream_t st) {
  auto* k = mix_real_kernel<KIND>;
  if (L.howmany <= 0) return cudaSuccess;
  const int smem = mix_smem_bytes(L.d);
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  const int64_t grid = (L.howmany + 2 * L.d.c - 1) / (2 * L.d.c);
  if (grid > 0x7fffffff) return cudaErrorInvalidValue;
  return launch_pdl(k, dim3(unsigned(grid)), dim3(L.d.nthr), size_t(smem), st, L);
}

}  // namespace plfft_b200
