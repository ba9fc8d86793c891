// Launch descriptors of the mixed-radix tile engine (mix.cuh), shared by the
// host planner (plan_mix.cpp) and the kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace plfft_b200 {

constexpr int kMixMaxStages = 8;
// Butterflies of radix R one thread holds at a time: as many as `budget`
// elements allow, so small radices keep as many loads in flight as large
// ones.  The budgets and launch bounds go together: FP32 pairs 12 elements
// at 80 registers, FP64 and the grouped kernel's single FP32 numbers 16 at
// 128 and 64.
constexpr int mix_held(int R, int budget) { return R >= budget ? 1 : budget / R; }
constexpr int kMixHeldPair = 12, kMixHeldSingle = 16;
constexpr int kMixThreadsPair = 768, kMixThreads64 = 512;  // resident threads per SM, largest CTA

// One radix stage of a tile of `c` transforms.  Butterfly j (< nb) of the
// stage is q = j / ns, r = j mod ns; it reads logical elements j + i nb and
// writes q ns R + r + i ns.  Between two stages the elements lie in shared
// memory in blocks of ns * R (the product of the radices done so far), each
// block followed by a pad that keeps the lanes of a warp on distinct banks;
// the reader's stride nb is a multiple of the block, so both sides stay
// linear in i.
struct MixStage {
  int radix, ns, nb, tw_off;
  int rpad;   // pad after each block of ns elements on the read side
  int rstep;  // address step of the inputs: nb + rpad * (nb / ns)
  int wblk;   // address of output block q: q * wblk  (ns * R + write-side pad)
  int total;  // butterflies of a full tile: c * nb
  uint32_t mul_nb, mul_ns;  // x / d = umulhi(x, mul) (0: d == 1)
};

struct MixDesc {
  int n, nstages;
  int c;        // engine elements (FP32: pairs of transforms, FP64: transforms) per tile
  int ld;       // shared-memory pitch of one of them, in 16-byte elements
  int nthr;     // threads per CTA
  int inplace;  // 1: one buffer, every middle stage held in registers at once; 0: two buffers
  int cf_in, cf_mid, cf_out;  // 1: consecutive threads take consecutive elements of the tile, 0: consecutive butterflies
  uint32_t mul_c;
  MixStage st[kMixMaxStages];
};

// element k of transform (member m, column col): base + m * mdist + col * cdist + k * kstride
struct MixAddr {
  int64_t mdist, cdist, kstride;
};

// two-level four-step twiddle W_N^e = lo[e mod 2^shift] * hi[e >> shift] on
// output k: e = column * k
template <class W>
struct MixPost {
  const W* lo;
  const W* hi;
  int shift;
};

// W: the twiddle type, float2 or double2
template <class W>
struct MixLaunch {
  const void* in;
  void* out;
  int64_t members;  // tiles = members * tpm
  int64_t ncols;    // transforms per member
  uint32_t tpm;     // tiles per member
  int wide_in, wide_out;  // FP32 pairs may be moved as aligned 16-byte words
  MixAddr ia, oa;
  double scale;
  const W* tw;
  MixPost<W> post;  // lo == nullptr: none
  MixDesc d;
  // share of shared memory, percent (0: the driver's choice); for the host, and
  // last, as d four bytes further on is loaded in smaller pieces (C2C n=11025 x
  // 1 12.4 us, 11.2 so)
  int carveout = 0;
};

// Real-data kinds (FusedRealKind) of N = 2M reals through a length-M tile
// (mix_real.cuh); distances in elements of each side's own type.
struct MixRealLaunch {
  const void* in;
  void* out;
  int64_t howmany, idist, odist;
  float scale;
  const float2* tw;
  const float2* post;
  const float2* rot;
  int wmode;                // adjoint weights, as RealFusedLaunch::wmode
  int pairs_in, pairs_out;  // the real side may be moved as aligned pairs
  uint32_t mul_half, mul_m;  // x / (M/2 + 1), x / M
  MixDesc d;                // n = M
};
bool mix_real_last_staged(int kind);
cudaError_t launch_mix_real(int kind, const MixRealLaunch& L, cudaStream_t st);

int mix_smem_bytes(const MixDesc& d);
cudaError_t launch_mix_f32(int dir, const MixLaunch<float2>& L, cudaStream_t st);
// the post twiddle goes by member, not by column
cudaError_t launch_mix_f32_members(int dir, const MixLaunch<float2>& L, cudaStream_t st);
// binary16 buffers; pairs: both aligned for 4-byte (re, im) accesses
cudaError_t launch_mix_f16(int dir, bool pairs, const MixLaunch<float2>& L, cudaStream_t st);
cudaError_t launch_mix_f16_scalar(int dir, const MixLaunch<float2>& L, cudaStream_t st);
cudaError_t launch_mix_f64(int dir, const MixLaunch<double2>& L, cudaStream_t st);

}  // namespace plfft_b200
