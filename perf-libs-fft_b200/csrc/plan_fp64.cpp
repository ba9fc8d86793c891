// FP64 plan nodes (kernels in fp64.cu).
//
// C2C: the mixed-radix tile engine (mix.cuh) in double for smooth on-chip n,
// direct sums for other n <= 4096, two mixed-radix passes for longer
// 7-smooth n = n1 n2 with both factors <= 4096.  R2C / C2R: the real data
// widened into a length-n complex sequence (Hermitian expansion for C2R),
// the C2C plan, then the half spectrum (or the real parts) extracted.
// Every table is computed in double on the host.
#include <cmath>
#include <sstream>

#include "plan.hpp"
#include "plan_mix.hpp"

namespace plfft_b200 {

namespace {

constexpr int kF64MaxOnChip = 4096;

bool smooth7(int64_t n) {
  for (int p : {2, 3, 5, 7})
    while (n % p == 0) n /= p;
  return n == 1;
}

double2 root64(int64_t k, int64_t n) {  // exp(-2 pi i k / n)
  double c, s;
  unit_root(k, n, c, s);
  return make_double2(c, -s);
}

// n two-pass (n = n1 n2, mixed-radix tiles) or, with n2 == 0, direct sums
struct F64C2CNode : Node {
  int64_t n = 0, n1 = 0, n2 = 0, chunk = 1;
  int dir = -1;
  Layout lay{};
  double scale = 1.0;
  MixLaunch<double2> p1{}, p2{};
  DevBuf tw1, tw2, lo, hi;
  size_t workspace() const override { return n2 ? size_t(chunk * n) * sizeof(double2) : 0; }
  bool reads_batch_first() const override { return n2 && chunk >= lay.howmany; }
  int launches() const override { return n2 ? int(2 * ((lay.howmany + chunk - 1) / chunk)) : 1; }
  cudaError_t run(const void* in, void* out, void* ws, cudaStream_t st) const override {
    const auto* x = static_cast<const double2*>(in);
    auto* y = static_cast<double2*>(out);
    if (!n2) {
      const F64DftLaunch L{x,          y,           lay.howmany, int(n), lay.istride, lay.idist,
                           lay.ostride, lay.odist, scale,       tw1.as<double2>()};
      return launch_fp64_dft(dir, L, st);
    }
    for (int64_t m0 = 0; m0 < lay.howmany; m0 += chunk) {
      MixLaunch<double2> a = p1, b = p2;
      a.members = b.members = std::min(chunk, lay.howmany - m0);
      a.in = x + m0 * lay.idist;
      a.out = ws;
      cudaError_t e = launch_mix_f64(dir, a, st);
      if (e != cudaSuccess) return e;
      b.in = ws;
      b.out = y + m0 * lay.odist;
      e = launch_mix_f64(dir, b, st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  std::string describe() const override {
    std::ostringstream o;
    o << "(c2c-fp64 n=" << n;
    if (n2)
      o << " four-step " << n1 << "x" << n2 << " chunk=" << chunk << " " << mix_describe(p1.d) << " "
        << mix_describe(p2.d);
    else
      o << " direct sums";
    o << ")";
    return o.str();
  }
};

struct F64RealNode : Node {
  std::unique_ptr<Node> c2c;  // length-n complex plan over a dense chunk
  F64RealLaunch base{};
  int64_t howmany = 1, chunk = 1;
  size_t work_bytes() const { return size_t(chunk * base.n) * sizeof(double2); }
  size_t workspace() const override { return (work_bytes() + 255) / 256 * 256 + c2c->workspace(); }
  bool reads_batch_first() const override { return chunk >= howmany; }
  int launches() const override { return int((howmany + chunk - 1) / chunk) * (2 + c2c->launches()); }
  cudaError_t run(const void* in, void* out, void* ws, cudaStream_t st) const override {
    F64RealLaunch L = base;
    L.in = in;
    L.out = out;
    L.work = static_cast<double2*>(ws);
    void* cws = static_cast<unsigned char*>(ws) + (work_bytes() + 255) / 256 * 256;
    for (int64_t m0 = 0; m0 < howmany; m0 += chunk) {
      const int64_t cnt = std::min(chunk, howmany - m0);
      if (cnt != chunk) return cudaErrorInvalidValue;  // chunk divides the batch (see make_fp64_node)
      cudaError_t e = launch_fp64_real(true, L, m0, cnt, st);
      if (e == cudaSuccess) e = c2c->run(L.work, L.work, cws, st);
      if (e == cudaSuccess) e = launch_fp64_real(false, L, m0, cnt, st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  std::string describe() const override {
    return std::string(base.c2r ? "(c2r" : "(r2c") + "-fp64 through complex n=" + std::to_string(base.n) + ") + " +
           c2c->describe();
  }
};

}  // namespace

std::unique_ptr<Node> make_fp64_c2c(int64_t n, const Layout& lay, int dir, double scale, std::string* why) {
  // 7-smooth n, and the 13-smooth ones the direct sums would take, but for the
  // shortest of these in batches that leave the chip idle: a short sum ends
  // before the long radix does (us, sums / engine: n=13 x 16 3.5 / 3.1, x 32
  // 3.5 / 4.1, x 1000 3.6 / 4.3, x 2000 3.7 / 4.0; n=26 x 64 4.1 / 4.3, x 1000
  // 4.2 / 4.5, x 2000 5.1 / 4.3; n=33 x 64 4.2 / 3.8)
  const bool sums = !smooth7(n) && n <= 26 && lay.howmany >= 32 && lay.howmany <= 1000;
  if (smooth7(n) || (is_smooth(n) && n <= kF64MaxOnChip && !sums))
    if (auto t = make_mix_c2c<double2>(n, lay, dir, scale, false, why)) return t;
  auto node = std::make_unique<F64C2CNode>();
  node->n = n;
  node->dir = dir;
  node->lay = lay;
  node->scale = scale;
  if (n <= kF64MaxOnChip) {
    std::vector<double2> tw(n);
    for (int64_t m = 0; m < n; ++m) tw[m] = root64(m, n);
    if (node->tw1.upload(tw) != cudaSuccess) return nullptr;
    return node;
  }
  if (!smooth7(n)) {
    if (why) *why = "FP64 on the device covers 7-smooth n, and other n <= 4096";
    return nullptr;
  }
  // four-step split with both factors on chip, n1 as close to sqrt(n) as possible
  int64_t best = 0;
  for (int64_t a = 2; a <= kF64MaxOnChip; ++a)
    if (n % a == 0 && n / a <= kF64MaxOnChip && (!best || std::llabs(a * a - n) < std::llabs(best * best - n))) best = a;
  if (!best) {
    if (why) *why = "FP64 length has no four-step split with factors <= 4096";
    return nullptr;
  }
  const int64_t n1 = node->n1 = best, n2 = node->n2 = n / best;
  node->chunk = std::max<int64_t>(1, std::min<int64_t>(lay.howmany, (int64_t(256) << 20) / (n * 16)));
  // pass 1: columns (member, n2 index) of length n1, times W_n^{col k};
  // pass 2: rows (member, n1 index) of length n2, written transposed
  if (!mix_shape(node->p1.d, n1, n2, true, true, 1, false) ||
      !mix_shape(node->p2.d, n2, n1, false, true, 1, false) ||
      node->tw1.upload(mix_twiddle_list<double2>(node->p1.d)) != cudaSuccess ||
      node->tw2.upload(mix_twiddle_list<double2>(node->p2.d)) != cudaSuccess)
    return nullptr;
  int shift = 0;
  while ((int64_t(1) << (2 * shift)) < n) ++shift;
  const int64_t L = int64_t(1) << shift;
  std::vector<double2> lo(L), hi((n + L - 1) / L);
  for (int64_t i = 0; i < L; ++i) lo[i] = root64(i, n);
  for (size_t i = 0; i < hi.size(); ++i) hi[i] = root64(int64_t(i) * L, n);
  if (node->lo.upload(lo) != cudaSuccess || node->hi.upload(hi) != cudaSuccess) return nullptr;
  auto pass = [](MixLaunch<double2>& m, int64_t ncols, MixAddr ia, MixAddr oa, double sc, const DevBuf& tw) {
    m.ncols = ncols;
    m.tpm = uint32_t((ncols + m.d.c - 1) / m.d.c);
    m.ia = ia;
    m.oa = oa;
    m.scale = sc;
    m.tw = tw.as<double2>();
  };
  pass(node->p1, n2, MixAddr{lay.idist, lay.istride, n2 * lay.istride}, MixAddr{n, 1, n2}, 1.0, node->tw1);
  pass(node->p2, n1, MixAddr{n, n2, 1}, MixAddr{lay.odist, lay.ostride, n1 * lay.ostride}, scale, node->tw2);
  node->p1.post = MixPost<double2>{node->lo.as<double2>(), node->hi.as<double2>(), shift};
  return node;
}

std::unique_ptr<Node> make_fp64_node(int kind, int64_t n, const Layout& lay, int dir, double scale,
                                     std::string* why) {
  if (kind == 0) return make_fp64_c2c(n, lay, dir, scale, why);
  if (kind != 1 && kind != 2) {
    if (why) *why = "FP64 real-to-real transforms have no device schedule";
    return nullptr;
  }
  auto node = std::make_unique<F64RealNode>();
  node->howmany = lay.howmany;
  // a chunk that divides the batch, of at most ~128 MB of complex workspace
  int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(lay.howmany, (int64_t(128) << 20) / (n * 16)));
  while (lay.howmany % chunk) --chunk;
  node->chunk = chunk;
  node->base = F64RealLaunch{nullptr, nullptr, nullptr, n, lay.istride, lay.idist, lay.ostride, lay.odist,
                             kind == 2 ? 1 : 0, scale};
  node->c2c = make_fp64_c2c(n, Layout{chunk, 1, n, 1, n}, kind == 2 ? 1 : -1, 1.0, why);
  if (!node->c2c) return nullptr;
  return node;
}

}  // namespace plfft_b200
