// Planner interface of the mixed-radix tile engine (plan_mix.cpp).
#pragma once
#include <memory>
#include <string>
#include <vector>

#include "mix.h"
#include "plan.hpp"

namespace plfft_b200 {

// radices 2..16 whose product is n, cheapest stage list first found; empty
// if n has a prime factor above 13
std::vector<int> mix_radices(int64_t n, int max_radix);
// instructions per element of that list's stages
double mix_stage_cost(int64_t n, int max_radix);
// radices, tile width, threads and buffers for length n and `count`
// transforms, `lanes` of them per engine element (FP32 2, FP64 1); c_req > 0
// asks for a tile width.  False: not on chip.
// staged: the last stage's results go to shared memory, not to the user's
// buffer.
bool mix_shape(MixDesc& d, int64_t n, int64_t count, bool cf_in, bool cf_out, int lanes, bool staged,
               int c_req = 0);
// stages and pads of length n (1: no stage), then a tile of exactly c such
// transforms for a CTA of `threads` threads and a shared-memory budget of
// max_elems 16-byte elements, any stage of which may run from shared memory to
// shared memory (false: does not fit)
bool mix_tile_layout(MixDesc& d, int n, int max_radix);
bool mix_tile_set(MixDesc& d, int c, int threads, int max_elems);
template <class V>
std::vector<V> mix_twiddle_list(const MixDesc& d);
// sets wide_in / wide_out from the buffers and addresses
void mix_wide(MixLaunch<float2>& L);
void mix_wide(MixLaunch<double2>& L);
std::string mix_describe(const MixDesc& d);

// one-pass C2C of a strided batch (half: binary16 buffers, V = float2);
// nullptr when n is not a supported on-chip length
template <class V>
std::unique_ptr<Node> make_mix_c2c(int64_t n, const Layout& lay, int dir, double scale, bool half, std::string* why);

// one-pass C2C of binary16 buffers; nullptr when n is not an on-chip length
std::unique_ptr<Node> make_half_c2c(int64_t n, const Layout& lay, int dir, double scale, std::string* why);
// one-pass real transform (FusedRealKind) of even n = 2M with on-chip smooth
// M, unit strides; nullptr otherwise
std::unique_ptr<Node> make_mix_real(int kind, int64_t n, const Layout& lay, float scale, int wmode);

}  // namespace plfft_b200
