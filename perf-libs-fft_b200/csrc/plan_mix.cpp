// Host planner of the mixed-radix tile engine (mix.cuh): radix list, shared
// memory layout and launch shape of an on-chip length.
#include "plan_mix.hpp"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <sstream>

namespace plfft_b200 {

namespace {

// Instructions a radix-R stage spends per element: the two shared-memory
// accesses, the twiddle load and product (14), the butterfly's index and
// address set-up spread over its R elements (60 / R), and the codelet.
double radix_cost(int R) {
  static const double codelet[17] = {0, 0,   1.0, 2.3, 2.0, 3.6, 3.7, 5.3, 3.6,
                                     5.0, 5.0, 8.5, 5.0, 10., 6.7, 6.5, 5.5};
  return 14.0 + 60.0 / R + codelet[R];
}

// cheapest non-increasing radix list of n; composite radices up to `cap`
// (the primes 11 and 13 always)
void search(int64_t n, int last, int cap, std::vector<int>& cur, double cost, std::vector<int>& best,
            double& best_cost) {
  if (n == 1) {
    if (best.empty() || cost < best_cost - 1e-9) {
      best = cur;
      best_cost = cost;
    }
    return;
  }
  if (int(cur.size()) >= kMixMaxStages) return;
  for (int R = int(std::min<int64_t>(last, n)); R >= 2; --R) {
    if (n % R || (R > cap && R != 11 && R != 13)) continue;
    cur.push_back(R);
    search(n / R, R, cap, cur, cost + radix_cost(R), best, best_cost);
    cur.pop_back();
  }
}

uint32_t magic(int d) { return d <= 1 ? 0u : uint32_t(((uint64_t(1) << 32) + uint64_t(d) - 1) / uint64_t(d)); }

// bank conflicts of one warp-wide access pattern: extra passes beyond the
// fewest, `eb`-byte elements (8 or 16) at addr(lane)
template <class F>
int conflicts(int eb, F addr) {
  const int lanes = 128 / eb;  // lanes served per pass
  int worst = 0;
  for (int base = 0; base < 32; base += lanes) {
    int count[16] = {0};
    int seen[32];
    int ns = 0;
    for (int l = base; l < base + lanes; ++l) {
      const int a = addr(l);
      if (a < 0) continue;
      bool dup = false;
      for (int k = 0; k < ns; ++k) dup = dup || seen[k] == a;
      if (dup) continue;
      seen[ns++] = a;
      ++count[a % lanes];
    }
    int mx = 1;
    for (int b = 0; b < lanes; ++b) mx = std::max(mx, count[b]);
    worst += mx - 1;
  }
  return worst;
}

}  // namespace

std::vector<int> mix_radices(int64_t n, int max_radix) {
  std::vector<int> cur, best;
  double bc = 0;
  search(n, 16, max_radix, cur, 0, best, bc);
  return best;
}

double mix_stage_cost(int64_t n, int max_radix) {
  double c = 0;
  for (int r : mix_radices(n, max_radix)) c += radix_cost(r);
  return c;
}

static bool mix_layout(MixDesc& d, const std::vector<int>& radices, int elem_bytes = 16) {
  const int n = d.n;
  d.nstages = int(radices.size());
  if (d.nstages < 1 || d.nstages > kMixMaxStages) return false;
  int ns = 1, tw = 0;
  for (int s = 0; s < d.nstages; ++s) {
    MixStage& st = d.st[s];
    st.radix = radices[s];
    st.ns = ns;
    st.nb = n / st.radix;
    st.tw_off = tw;
    st.mul_nb = magic(st.nb);
    st.mul_ns = magic(ns);
    st.rpad = 0;
    if (ns > 1) tw += (st.radix - 1) * ns;
    ns *= st.radix;
  }
  // pad of each exchange: fewest conflicts over a few warps of the writer
  // and the reader, lanes along j; the smallest such pad
  int ld = n;
  for (int s = 0; s + 1 < d.nstages; ++s) {
    MixStage& w = d.st[s];
    MixStage& r = d.st[s + 1];
    const int block = w.ns * w.radix;
    int best_pad = 0, best_c = -1;
    for (int pad = 0; pad < 128 / elem_bytes; ++pad) {
      if (pad > 1 && pad * 4 > block) break;  // a quarter more shared memory at most
      int c = 0;
      for (int w0 = 0; w0 < 4; ++w0) {
        const int j0 = w0 * 32 * 3;
        c += conflicts(elem_bytes, [&](int l) {
          const int j = j0 + l;
          if (j >= w.nb) return -1;
          return (j / w.ns) * (block + pad) + j % w.ns;
        });
        c += conflicts(elem_bytes, [&](int l) {
          const int j = j0 + l;
          if (j >= r.nb) return -1;
          return j + pad * (j / block);
        });
      }
      if (best_c < 0 || c < best_c) {
        best_c = c;
        best_pad = pad;
      }
    }
    w.wblk = block + best_pad;
    r.rpad = best_pad;
    r.rstep = r.nb + best_pad * (r.nb / block);
    ld = std::max(ld, n + best_pad * (n / block));
  }
  d.st[0].rstep = d.st[0].nb;
  d.st[d.nstages - 1].wblk = n;
  if (d.nstages == 1) d.st[0].wblk = n;
  d.ld = ld | 1;  // odd: lanes along the transforms of a tile do not collide
  return true;
}

// `c` transforms per tile of an already laid out length
static void mix_set_tile(MixDesc& d, int c) {
  d.c = c;
  d.mul_c = magic(c);
  for (int s = 0; s < d.nstages; ++s) d.st[s].total = c * d.st[s].nb;
}

namespace {

int sm_count() {
  static const int n = [] {
    int dev = 0, sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
                   cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0
               ? sms
               : 148;  // no device here (the planner's own tests)
  }();
  return n;
}

// shared memory of an SM that tiles may fill, and of one CTA
constexpr int kSmemPerSm = 227 * 1024, kSmemPerCta = 224 * 1024;
// Estimated time of a shape per element, in issued instructions: every
// stage's issue work with idle warps' share, spread over the resident
// threads that hide its latency.
double shape_cost(const MixDesc& d, int64_t ncols, int lanes) {
  const int resident = lanes == 2 ? kMixThreadsPair : kMixThreads64;
  const int held = lanes == 2 ? kMixHeldPair : kMixHeldSingle;
  const int64_t bytes = int64_t(d.c) * d.ld * 16 * (d.inplace ? 1 : 2);
  if (bytes > kSmemPerCta) return -1;
  const int per_sm =
      int(std::min<int64_t>({int64_t(resident / d.nthr), int64_t(kSmemPerSm) / (bytes + 1024), 32}));
  if (per_sm < 1) return -1;
  double work = 0;
  const int warps = d.nthr / 32;
  for (int s = 0; s < d.nstages; ++s) {
    const MixStage& st = d.st[s];
    const int nb = mix_held(st.radix, held);
    const int64_t per_iter = int64_t(nb) * d.nthr;
    const int64_t iters = (st.total + per_iter - 1) / per_iter;
    // butterflies issued (whole warps), plus the idle ones' index work
    const double issued = double((st.total + 31) / 32);
    const double idle = double(iters * nb * warps) - issued;
    work += issued * st.radix * radix_cost(st.radix) + idle * 25.0 + iters * warps * 40.0;
  }
  const int64_t tiles = (ncols + d.c - 1) / d.c;
  const double used = double(ncols) / double(tiles * d.c);  // a ragged last tile
  double cost = work * 32.0 / (double(d.c) * d.n * used);
  // fewer resident warps, or few resident CTAs (their barriers stop a large
  // share of the SM), leave latency exposed: N=1000 x 16384 FP32 61.9 us with
  // six CTAs of 128 threads, 65.5 with three of 256, 96 with one of 416
  cost *= 1.0 + 0.5 * (1.0 - std::min(1.0, per_sm * d.nthr / double(resident))) + 1.0 / per_sm;
  // a second buffer takes shared memory from the L1 that serves the twiddles
  // (N=500 x 32768: 59.5 us with one buffer, 71 with two)
  if (!d.inplace) cost *= 1.12;
  // too few tiles for the chip: the tile's own latency counts
  const double waves = double(tiles) / (double(sm_count()) * per_sm);
  if (waves < 1.0) cost *= 1.0 + 0.15 * (1.0 - waves) * double(d.c) * d.n / (16.0 * d.nthr);
  return cost;
}

}  // namespace

bool mix_shape(MixDesc& d, int64_t n, int64_t count, bool cf_in, bool cf_out, int lanes, bool staged, int c_req) {
  const int64_t ncols = (count + lanes - 1) / lanes;
  const int max_thr = lanes == 2 ? kMixThreadsPair : kMixThreads64;
  const int held = lanes == 2 ? kMixHeldPair : kMixHeldSingle;
  if (n < 2 || n > 16384) return false;
  std::vector<int> radices = mix_radices(n, 16);
  if (radices.empty()) return false;
  // A single stage gives a whole transform to one thread, and at 14 points and
  // more a dense side pays for lanes that lie n elements apart: two stages
  // (us, 2^22 numbers, one / two: C2C n=14 22.6 / 19.8, 15 23.3 / 15.7, 16
  // 28.2 / 16.8; C2R n=32 47.0 / 13.0; n=12 19.3 / 16.1, but its real kinds
  // of 1000 members 4.3 / 5.6).  Few members end sooner in one (C2C n=16 x 4
  // after another kernel 4.0 / 4.8, x 1000 4.9 / 4.3).
  if (n >= 14 && count > 128 && radices.size() == 1 && !(cf_in && cf_out)) radices = mix_radices(n, int(n) - 1);
  MixDesc best{};
  double best_cost = -1;
  // strided batches move segments of c consecutive elements: whole 32-byte
  // sectors at least, 64 or 128 bytes where the tile fits
  const int seg = (cf_in || cf_out) ? 4 : 1;
  const int cs[] = {1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16, 20, 24, 28, 32, 40, 48, 56, 64, 80, 96, 112, 128, 160, 192, 224, 256};
  MixDesc laid{};
  laid.n = int(n);
  laid.cf_in = cf_in;
  laid.cf_out = cf_out;
  if (!mix_layout(laid, radices)) return false;
  for (int c : cs) {
    if (c_req > 0 ? c != c_req : (c > 1 && int64_t(c) * n > 4096)) continue;
    if (c > ncols) break;
    MixDesc t = laid;
    mix_set_tile(t, c);
    for (int thr = 32; thr <= max_thr; thr += 32) {
      int need = 0;  // threads that hold every middle stage at once
      for (int s = 1; s < t.nstages - (staged ? 0 : 1); ++s) {
        const int nb = mix_held(t.st[s].radix, held);
        need = std::max(need, (t.st[s].total + nb - 1) / nb);
      }
      for (int ip = 0; ip < 2; ++ip) {
        if (ip ? need > thr : (t.nstages == 2 && !staged)) continue;
        t.nthr = thr;
        t.inplace = ip;  // two stages: one exchange, one buffer
        double cost = shape_cost(t, ncols, lanes);
        if (cost < 0) continue;
        if (seg > 1 && c < seg) cost *= 1.0 + 0.35 * (double(seg) / c - 1.0);
        if (best_cost < 0 || cost < best_cost) {
          best_cost = cost;
          best = t;
        }
      }
    }
  }
  if (best_cost < 0) return false;
  d = best;
  d.cf_mid = (cf_in && cf_out && d.c >= 8) ? 1 : 0;
  return true;
}

bool mix_tile_layout(MixDesc& d, int n, int max_radix) {
  d = MixDesc{};
  d.n = n;
  d.ld = 1;
  if (n == 1) return true;  // no stage: a copy
  const std::vector<int> radices = mix_radices(n, max_radix);
  return !radices.empty() && mix_layout(d, radices, int(sizeof(float2)));
}

bool mix_tile_set(MixDesc& d, int c, int threads, int max_elems) {
  d.nthr = threads;
  mix_set_tile(d, c);
  bool held = true;  // every stage may run as a middle stage here
  for (int s = 0; s < d.nstages; ++s)
    held = held && d.st[s].total <= int64_t(mix_held(d.st[s].radix, kMixHeldSingle)) * threads;
  d.inplace = held;
  return int64_t(c) * d.ld * (held ? 1 : 2) <= max_elems;
}

template <class V>
struct MixTypes;
template <>
struct MixTypes<float2> {
  using S = float;
};
template <>
struct MixTypes<double2> {
  using S = double;
};

// stage twiddles, stage by stage: row i = 1..R-1, entry r: exp(-2 pi i r i / (ns R))
template <class V>
std::vector<V> mix_twiddle_list(const MixDesc& d) {
  using S = typename MixTypes<V>::S;
  std::vector<V> tw;
  for (int s = 1; s < d.nstages; ++s) {
    const MixStage& st = d.st[s];
    for (int i = 1; i < st.radix; ++i)
      for (int r = 0; r < st.ns; ++r) {
        double c, sn;
        unit_root(int64_t(r) * i, int64_t(st.ns) * st.radix, c, sn);
        V v;
        v.x = S(c);
        v.y = S(-sn);
        tw.push_back(v);
      }
  }
  if (tw.empty()) tw.push_back(V{});
  return tw;
}
template std::vector<float2> mix_twiddle_list<float2>(const MixDesc&);
template std::vector<double2> mix_twiddle_list<double2>(const MixDesc&);

void mix_wide(MixLaunch<float2>& L) {
  auto ok = [](const void* p, const MixAddr& a) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && a.cdist == 1 && a.kstride % 2 == 0 && a.mdist % 2 == 0;
  };
  L.wide_in = ok(L.in, L.ia);
  L.wide_out = ok(L.out, L.oa);
}
void mix_wide(MixLaunch<double2>&) {}

std::string mix_describe(const MixDesc& d) {
  std::ostringstream o;
  o << "mix n=" << d.n << " c=" << d.c << " threads=" << d.nthr << (d.inplace ? " one-buffer" : " two-buffers")
    << " radices=";
  for (int i = 0; i < d.nstages; ++i) o << (i ? "x" : "") << d.st[i].radix;
  return o.str();
}

namespace {

template <class V>
struct MixNode : Node {
  MixLaunch<V> base{};
  int dir = -1;
  bool half = false;
  DevBuf tw;
  cudaError_t run(const void* in, void* out, void*, cudaStream_t st) const override {
    MixLaunch<V> L = base;
    L.in = in;
    L.out = out;
    mix_wide(L);
    if constexpr (sizeof(V) == 16)
      return launch_mix_f64(dir, L, st);
    else
      return half ? launch_mix_f16(dir, (reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % 4 == 0, L, st)
                  : launch_mix_f32(dir, L, st);
  }
  std::string describe() const override {
    return std::string("(c2c-") + (sizeof(V) == 16 ? "fp64 " : (half ? "fp16 " : "")) + mix_describe(base.d) + ")";
  }
};

}  // namespace

template <class V>
std::unique_ptr<Node> make_mix_c2c(int64_t n, const Layout& lay, int dir, double scale, bool half, std::string* why) {
  auto node = std::make_unique<MixNode<V>>();
  // strided batches whose members interleave: consecutive lanes take
  // consecutive members
  const bool cf_in = lay.howmany > 1 && lay.istride > 1 && std::llabs(lay.idist) < lay.istride;
  const bool cf_out = lay.howmany > 1 && lay.ostride > 1 && std::llabs(lay.odist) < lay.ostride;
  int creq = 0;
  if (const char* v = std::getenv("PLFFT_B200_MIX_C")) creq = std::max(0, std::atoi(v));
  MixDesc& d = node->base.d;
  if (!mix_shape(d, n, lay.howmany, cf_in, cf_out, sizeof(V) == 16 ? 1 : 2, false, creq) &&
      !(creq && mix_shape(d, n, lay.howmany, cf_in, cf_out, sizeof(V) == 16 ? 1 : 2, false)))
    return nullptr;
  if (node->tw.upload(mix_twiddle_list<V>(d)) != cudaSuccess) {
    if (why) *why = "device allocation failed";
    return nullptr;
  }
  node->dir = dir;
  node->half = half;
  node->base.members = 1;
  node->base.ncols = lay.howmany;
  const int64_t per_tile = int64_t(d.c) * (sizeof(V) == 16 ? 1 : 2);
  node->base.tpm = uint32_t((lay.howmany + per_tile - 1) / per_tile);
  node->base.ia = MixAddr{0, lay.idist, lay.istride};
  node->base.oa = MixAddr{0, lay.odist, lay.ostride};
  node->base.scale = scale;
  node->base.tw = node->tw.template as<V>();
  node->base.post = MixPost<V>{nullptr, nullptr, 0};
  return node;
}
template std::unique_ptr<Node> make_mix_c2c<float2>(int64_t, const Layout&, int, double, bool, std::string*);
template std::unique_ptr<Node> make_mix_c2c<double2>(int64_t, const Layout&, int, double, bool, std::string*);

namespace {

// binary16 power of two: compile-time stages
struct Pow2HalfNode : Node {
  int n = 0, dir = -1;
  Pow2HalfLaunch base{};
  DevBuf tw;
  cudaError_t run(const void* in, void* out, void*, cudaStream_t st) const override {
    Pow2HalfLaunch L = base;
    L.pairs = (reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % 4 == 0;
    L.in = in;
    L.out = out;
    return launch_c2c_pow2_half(n, dir, L, st);
  }
  std::string describe() const override {
    return "(c2c-fp16 pow2 n=" + std::to_string(n) + " e=" + std::to_string(pow2_half_e(n)) + ")";
  }
};

}  // namespace

std::unique_ptr<Node> make_half_c2c(int64_t n, const Layout& lay, int dir, double scale, std::string* why) {
  // dense powers of two: 7.8 us against 17 us of the tile engine at N=1024 x
  // 4096 (33.5 MB), 6.7 us at N=256 x 16384
  if (n < 64 || n > 8192 || (n & (n - 1)) || lay.istride != 1 || lay.ostride != 1)
    return make_mix_c2c<float2>(n, lay, dir, scale, true, why);
  auto node = std::make_unique<Pow2HalfNode>();
  node->n = int(n);
  node->dir = dir;
  const int e = pow2_half_e(n);
  std::vector<int> radices;
  int64_t rest = n;
  int ke = 0;
  for (; rest % e == 0 && rest > 1; rest /= e) ++ke;
  if (rest > 1) radices.push_back(int(rest));
  radices.insert(radices.end(), ke, e);
  std::vector<float2> tw;
  make_desc(int(n), radices, tw);
  if (node->tw.upload(tw) != cudaSuccess) {
    if (why) *why = "device allocation failed";
    return nullptr;
  }
  node->base.howmany = lay.howmany;
  node->base.idist = lay.idist;
  node->base.odist = lay.odist;
  node->base.scale = float(scale);
  node->base.tw = node->tw.as<float2>();
  return node;
}

namespace {

struct MixRealNode : Node {
  int kind = 0;
  MixRealLaunch base{};
  DevBuf tab;
  cudaError_t run(const void* in, void* out, void*, cudaStream_t st) const override {
    MixRealLaunch L = base;
    L.in = in;
    L.out = out;
    L.pairs_in = reinterpret_cast<uintptr_t>(in) % 8 == 0 && (L.howmany == 1 || L.idist % 2 == 0);
    L.pairs_out = reinterpret_cast<uintptr_t>(out) % 8 == 0 && (L.howmany == 1 || L.odist % 2 == 0);
    return launch_mix_real(kind, L, st);
  }
  std::string describe() const override {
    static const char* names[] = {"r2c",  "c2r",  "dct2", "dst2", "dct3", "dst3",
                                  "dct4", "dst4", "r2hc", "hc2r", "dht"};
    return std::string("(") + names[kind] + "-half n=" + std::to_string(2 * base.d.n) + " one pass " +
           mix_describe(base.d) + ")";
  }
};

}  // namespace

std::unique_ptr<Node> make_mix_real(int kind, int64_t n, const Layout& lay, float scale, int wmode) {
  if (n % 2 || n < 4 || lay.istride != 1 || lay.ostride != 1) return nullptr;
  const int64_t m = n / 2;
  auto node = std::make_unique<MixRealNode>();
  MixDesc& d = node->base.d;
  int creq = 0;
  if (const char* v = std::getenv("PLFFT_B200_MIX_C")) creq = std::max(0, std::atoi(v));
  const bool staged = mix_real_last_staged(kind);
  if (!mix_shape(d, m, lay.howmany, false, false, 2, staged, creq) &&
      !(creq && mix_shape(d, m, lay.howmany, false, false, 2, staged)))
    return nullptr;
  std::vector<float2> tab = mix_twiddle_list<float2>(d);
  const bool iv = kind == FR_DCT4 || kind == FR_DST4;
  const size_t post_off = tab.size();
  for (int64_t k = 0; k <= m; ++k) {  // W_N^k; DCT-IV / DST-IV: exp(i pi k / N) = W_{2N}^{-k}
    double c, s;
    unit_root(iv ? 2 * k : k, iv ? 4 * n : n, c, s);
    tab.push_back(make_float2(float(c), float(iv ? s : -s)));
  }
  const size_t rot_off = tab.size();
  for (int64_t k = 0; k <= m; ++k) {  // exp(-i pi k / 2N) = W_{4N}^k; DCT-IV / DST-IV: exp(i pi (4k+1) / 4N)
    double c, s;
    unit_root(iv ? 4 * k + 1 : k, iv ? 8 * n : 4 * n, c, s);
    tab.push_back(make_float2(float(c), float(iv ? s : -s)));
  }
  if (node->tab.upload(tab) != cudaSuccess) return nullptr;
  node->kind = kind;
  MixRealLaunch& L = node->base;
  L.howmany = lay.howmany;
  L.idist = lay.idist;
  L.odist = lay.odist;
  L.scale = scale;
  L.tw = node->tab.as<float2>();
  L.post = L.tw + post_off;
  L.rot = L.tw + rot_off;
  L.wmode = wmode;
  L.mul_half = magic(int(m / 2 + 1));
  L.mul_m = magic(int(m));
  return node;
}

}  // namespace plfft_b200
