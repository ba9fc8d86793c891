// Persistent grouped kernel: thousands of C2C FP32 transforms of mixed
// length in one launch per dependency phase.
//
// A group (grouped_plan.cpp) is a list of tasks.  Every task is one of:
//   GT_TILE   : `cnt` transforms (or four-step columns/rows) of one on-chip
//               length, element (c, k) at base + c*cdist + k*kstride, with an
//               optional prologue op on the loaded values and an optional
//               epilogue op on the results;
//   GT_RADER  : a whole Rader transform of prime length P, P-1 on chip;
//   GT_BLUE   : a whole Bluestein transform whose length-M convolution fits
//               on chip.
// Lengths that do not fit on chip become four-step tiles in two phases (and
// Rader/Bluestein convolutions of such lengths in four).  CTAs are resident
// for the whole phase and take tasks from a device counter in order of
// decreasing cost; the last CTA to finish resets the counter, so a captured
// CUDA graph can be replayed.
//
// This replaces, for mixed batches, the one-plan-per-length execution a
// PLFFT user would otherwise run (a plan per length, reference
// src/plfft.cpp:427-517 and the batched plan of src/batched_1d_plan.hpp).
#include "kernels.h"
#include "mix.cuh"
#include "ptx.cuh"

namespace plfft_b200 {

// The on-chip transforms run the stages of the mixed-radix engine (mix.cuh)
// with the stage list of the task in shared memory.  256 threads at 64
// registers and 36 KB of tile, four CTAs per SM: while some tiles wait for
// their loads or at a barrier the others compute (two CTAs of 512 threads
// took 807 us on the 4000-transform mix, these 727, and 659 with the lengths
// and splits that grouped_plan.cpp chooses by cost), and 16 four-step columns
// of 256 are whole 128-byte segments.
constexpr int kGroupThreads = 256, kGroupPerSm = 4;

__device__ __forceinline__ float2 group_conj(float2 v, bool on) { return on ? make_float2(v.x, -v.y) : v; }

// plain loads and stores of a tile; a backward tile is the conjugate of the
// forward transform of the conjugated input, so one set of stages serves both
struct GroupIo {
  const GTask* T;
  const float2* in;
  float2* out;
  bool conj;

  template <int R>
  __device__ __forceinline__ void load(int c, int j, int nb, float2 (&x)[R]) const {
    const float2* p = in + int64_t(c) * T->icdist + int64_t(j) * T->ikstride;
    const int64_t step = int64_t(nb) * T->ikstride;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      x[i] = group_conj(*p, conj);
      p += step;
    }
  }
  template <int R>
  __device__ __forceinline__ void store(int c, int k, int kstep, float2 (&x)[R]) const {
    float2* p = out + int64_t(c) * T->ocdist + int64_t(k) * T->okstride;
    const int64_t step = int64_t(kstep) * T->okstride;
    const bool tw = T->post_op == GO_TWIDDLE;
    const float s = T->scale;
    const uint32_t col = uint32_t(T->col0) + uint32_t(c);
    const int shift = T->tw2_shift;
    const float2* lo = T->tw2.lo;
    const float2* hi = T->tw2.hi;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float2 y = x[i];  // a backward tile's twiddle is conj(W): conj(y W) = conj(y) conj(W)
      if (tw) {
        const uint32_t e = col * uint32_t(k + i * kstep);
        y = cmul(y, cmul(__ldg(lo + (e & ((1u << shift) - 1u))), __ldg(hi + (e >> shift))));
      }
      *p = cscale(group_conj(y, conj), s);
      p += step;
    }
  }
};

// middle stages [first, last) of the tile in `src`; returns the buffer that
// holds the result
__device__ __forceinline__ float2* group_stages(const MixDesc& d, const float2* tw, float2* src, float2* dst,
                                                const GroupIo& io, int cnt, int first, int last) {
  for (int si = first; si < last; ++si) {
    mix_dispatch<float2, -1, MIX_MID>(d, si, tw, src, dst, io, cnt);
    __syncthreads();
    float2* t = src;
    src = dst;
    dst = t;
  }
  return src;
}

__device__ void run_tile(const GTask& T, const MixDesc& d, const GroupPhase& P, float2* sm) {
  const int n = T.n, cnt = T.cnt, ld = d.ld;
  GroupIo io;
  io.T = &T;
  io.in = P.bases[T.in_buf] + T.in_off;
  io.out = P.bases[T.out_buf] + T.out_off;
  io.conj = T.dir > 0;
  const float2* tw = P.tws[T.desc];
  float2* src = sm;
  float2* dst = d.inplace ? sm : sm + d.c * ld;
  const int ns = d.nstages;
  if (ns == 0) {  // length 1: a copy
    for (int c = threadIdx.x; c < cnt; c += blockDim.x)
      io.out[int64_t(c) * T.ocdist] = cscale(io.in[int64_t(c) * T.icdist], T.scale);
    return;
  }
  int first = 1;
  if (T.pre_op == GO_NONE) {
    mix_dispatch<float2, -1, MIX_FIRST>(d, 0, tw, src, src, io, cnt);
    __syncthreads();
  } else {
    // gathered or chirped inputs of a long convolution, staged in order; the
    // convolution's forward transform, so no conjugation
    first = 0;
    const bool kfast = T.pre_op == GO_GATHER;
    for (int f = threadIdx.x; f < cnt * n; f += blockDim.x) {
      const int c = kfast ? f / n : f % cnt, k = kfast ? f - c * n : f / cnt;
      const int64_t e = T.ie0 + int64_t(c) * T.iec + int64_t(k) * T.iek;
      float2 v = make_float2(0.f, 0.f);
      if (T.pre_op == GO_GATHER)
        v = io.in[int64_t(T.perm_in[e]) * T.ikstride];
      else if (e < T.pre_len)
        v = cmul(io.in[int64_t(c) * T.icdist + int64_t(k) * T.ikstride], T.pre_tab[e]);
      src[c * ld + k] = v;
    }
    __syncthreads();
  }
  if ((T.post_op == GO_NONE || T.post_op == GO_TWIDDLE) && ns > 1) {
    float2* at = group_stages(d, tw, src, dst, io, cnt, first, ns - 1);
    mix_dispatch<float2, -1, MIX_LAST>(d, ns - 1, tw, at, at, io, cnt);
    return;
  }
  const float2* z = group_stages(d, tw, src, dst, io, cnt, first, ns);
  const float2* xin = P.bases[T.aux_buf] + T.aux_off;
  const bool kfast = T.okstride == 1 || T.post_op == GO_SCATTER;
  for (int f = threadIdx.x; f < cnt * n; f += blockDim.x) {
    const int c = kfast ? f / n : f % cnt, k = kfast ? f - c * n : f / cnt;
    float2 y = group_conj(z[c * ld + k], io.conj);
    const int64_t e = T.oe0 + int64_t(c) * T.oec + int64_t(k) * T.oek;  // logical output index
    switch (T.post_op) {
      case GO_TWIDDLE: {
        const uint32_t q = (uint32_t(T.col0) + uint32_t(c)) * uint32_t(k);
        const float2 w = cmul(__ldg(T.tw2.lo + (q & ((1u << T.tw2_shift) - 1u))), __ldg(T.tw2.hi + (q >> T.tw2_shift)));
        y = io.conj ? cmulc(y, w) : cmul(y, w);
        break;
      }
      case GO_SPEC_SAVE0:
        if (e == 0) T.sum0[0] = y;
        y = cmul(y, T.post_tab[e]);
        break;
      case GO_SPEC:
        y = cmul(y, T.post_tab[e]);
        break;
      case GO_CHIRP:
        if (e >= T.post_len) continue;
        y = cmul(y, T.post_tab[e]);
        break;
      case GO_SCATTER: {
        const float2 x0 = xin[0];
        io.out[int64_t(T.perm_out[e]) * T.okstride] = cscale(cadd(x0, y), T.scale);
        if (e == 0) io.out[0] = cscale(cadd(x0, T.sum0[0]), T.scale);
        continue;
      }
      default: break;
    }
    io.out[int64_t(c) * T.ocdist + int64_t(k) * T.okstride] = cscale(y, T.scale);
  }
}

// whole Rader (prime P, P - 1 = T.n on chip) or Bluestein transform (length
// T.pre_len, convolution length T.n on chip)
template <bool RADER>
__device__ void run_conv(const GTask& T, const MixDesc& d, const GroupPhase& P, float2* sm) {
  const int m = T.n;
  GroupIo io;
  io.T = &T;
  io.in = P.bases[T.in_buf] + T.in_off;
  io.out = P.bases[T.out_buf] + T.out_off;
  io.conj = false;
  const float2* tw = P.tws[T.desc];
  float2* other = d.inplace ? sm : sm + d.ld;
  __shared__ float2 a0;
  for (int q = threadIdx.x; q < m; q += blockDim.x) {
    float2 v = make_float2(0.f, 0.f);
    if (RADER)
      v = io.in[int64_t(T.perm_in[q]) * T.ikstride];
    else if (q < T.pre_len)
      v = cmul(io.in[int64_t(q) * T.ikstride], T.pre_tab[q]);
    sm[q] = v;
  }
  __syncthreads();
  float2* z = group_stages(d, tw, sm, other, io, 1, 0, d.nstages);
  // the product, conjugated: the inverse transform is the conjugate of the
  // forward one of it
  const float2* spec = RADER ? T.post_tab : T.post_tab2;
  for (int q = threadIdx.x; q < m; q += blockDim.x) {
    const float2 v = z[q];
    if (RADER && q == 0) a0 = v;
    z[q] = group_conj(cmul(v, spec[q]), true);
  }
  __syncthreads();
  z = group_stages(d, tw, z, z == sm ? other : sm, io, 1, 0, d.nstages);
  if (RADER) {
    const float2 x0 = io.in[0];
    for (int q = threadIdx.x; q < m; q += blockDim.x)
      io.out[int64_t(T.perm_out[q]) * T.okstride] = cscale(cadd(x0, group_conj(z[q], true)), T.scale);
    if (threadIdx.x == 0) io.out[0] = cscale(cadd(x0, a0), T.scale);
  } else {
    for (int k = threadIdx.x; k < T.pre_len; k += blockDim.x)
      io.out[int64_t(k) * T.okstride] = cscale(cmul(group_conj(z[k], true), T.pre_tab[k]), T.scale);
  }
}

__global__ void __launch_bounds__(kGroupThreads, kGroupPerSm) grouped_kernel(const GroupPhase P) {
  extern __shared__ float2 smem[];
  // tasks in hand: the current one and the next, whose description is on its
  // way to shared memory while the current one runs, as is the index of the
  // one after it (fetched one after the other they cost 2 us a task)
  __shared__ GTask hand[2];
  __shared__ int index[2];
  static_assert(sizeof(GTask) % 8 == 0, "copied eight bytes at a time");
  auto fetch = [&](int slot, int t) {
    if (t >= P.ntasks) return;
    const unsigned char* from = reinterpret_cast<const unsigned char*>(P.tasks + t);
    unsigned char* to = reinterpret_cast<unsigned char*>(&hand[slot]);
    for (int i = 8 * threadIdx.x; i < int(sizeof(GTask)); i += 8 * blockDim.x) cp_async8(to + i, from + i);
  };
  // the first task is the CTA's own, the others come from the counter
  if (threadIdx.x == 0) {
    index[0] = blockIdx.x;
    index[1] = gridDim.x + atomicAdd(P.counter, 1);
  }
  __syncthreads();
  fetch(0, index[0]);
  cp_async_wait_all();
  __syncthreads();
  for (int slot = 0;; slot ^= 1) {
    if (index[slot] >= P.ntasks) break;
    fetch(slot ^ 1, index[slot ^ 1]);
    int after = 0;
    if (threadIdx.x == 0) after = gridDim.x + atomicAdd(P.counter, 1);
    __syncthreads();  // index[slot] is read by all before it is replaced below
    const GTask& T = hand[slot];
    switch (T.type) {
      case GT_TILE: run_tile(T, T.d, P, smem); break;
      case GT_RADER: run_conv<true>(T, T.d, P, smem); break;
      case GT_BLUE: run_conv<false>(T, T.d, P, smem); break;
      default: break;
    }
    cp_async_wait_all();
    if (threadIdx.x == 0) index[slot] = after;
    __syncthreads();
  }
  // the last CTA out resets the counters for the next launch / graph replay
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(P.done, 1) == int(gridDim.x) - 1) {
      *P.counter = 0;
      *P.done = 0;
      __threadfence();
    }
  }
}

int group_threads() { return kGroupThreads; }
int group_max_smem_elems() { return 36 * 1024 / int(sizeof(float2)); }
// one CTA per SM, less the task descriptions
int group_most_smem_elems() { return 220 * 1024 / int(sizeof(float2)); }

cudaError_t launch_grouped(const GroupPhase& P, int grid, int smem_bytes, cudaStream_t st) {
  const cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_kernel), smem_bytes);
  if (e != cudaSuccess) return e;
  grouped_kernel<<<grid, kGroupThreads, smem_bytes, st>>>(P);
  return cudaGetLastError();
}

int grouped_blocks_per_sm(int smem_bytes) {
  int per = 0;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(grouped_kernel), smem_bytes) == cudaSuccess)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, grouped_kernel, kGroupThreads, smem_bytes);
  return per < 1 ? 1 : per;
}

}  // namespace plfft_b200
