// owl_tables.hpp -- host-side tables for one (E, W, H) shape: twiddles, the
// IBDWT weights factored per column and per line, and the big-word data.
//
// Word model (reference src/state.h:14-17): N = 2 W H words, step = N - E mod N,
// extra(k) = step k mod N, word k is big (one more bit) iff extra(k) < E mod N,
// weight(k) = 2^(extra(k)/N) (src/Gpu.cpp:42-56). Complex element j = j2 + H j1
// (line j2, column j1) holds words 2j and 2j+1 (src/Gpu.cpp:40 kAt), so
// extra(2j+e) = (X1[j1] + X2[2 j2 + e]) mod N with X1 = step 2H j1 mod N and
// X2 = step (2 j2 + e) mod N; the weight is the product of the two table
// factors, halved when X1 + X2 >= N.
//
// Twiddles are evaluated in long double after an exact octant reduction of the
// angle and rounded once to double (the reference builds its tables in long
// double too, src/TrigBufCache.cpp:22-120).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <stdexcept>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

#include "owl_dft.cuh"

namespace owl {

struct HostC {
  double x, y;
};

// cos and sin of 2 pi k / n
inline void root_ld(uint64_t n, uint64_t k, long double* c, long double* s) {
  const long double PI_L = 3.141592653589793238462643383279502884L;
  uint64_t q = 8 * n, p = 8 * (k % n);
  bool negS = false, negC = false, swp = false;
  if (2 * p > q) { p = q - p; negS = true; }
  if (4 * p > q) { p = q / 2 - p; negC = true; }
  if (8 * p > q) { p = q / 4 - p; swp = true; }
  long double a = 2.0L * PI_L * (long double)p / (long double)q;
  long double cc = cosl(a), ss = sinl(a);
  if (swp) { std::swap(cc, ss); }
  if (negC) { cc = -cc; }
  if (negS) { ss = -ss; }
  *c = cc;
  *s = ss;
}

// forward root w_n^k = exp(-2 pi i k / n)
inline HostC root(uint64_t n, uint64_t k) {
  long double c, s;
  root_ld(n, k, &c, &s);
  return HostC{(double)c, (double)-s};
}

// Many roots of one order n (a multiple of 8): w_n^k as a product of two tabulated factors, taken in long
// double and rounded once (sine and cosine of every entry would make the line groups' records the longest
// part of making a plan: 100K roots at 8M words). The factors, rounded, are the kernels' two-level table.
class Roots {
 public:
  explicit Roots(uint32_t n) : n8_(n / 8) {
    while ((1ull << (2 * sh_)) < n) { ++sh_; }
    lo_.resize(1u << sh_);
    hi_.resize((n - 1) / (1u << sh_) + 1);
    for (uint32_t i = 0; i < lo_.size(); ++i) { root_ld(n, i, &lo_[i].first, &lo_[i].second); }
    for (uint32_t i = 0; i < hi_.size(); ++i) { root_ld(n, (uint64_t)i << sh_, &hi_[i].first, &hi_[i].second); }
    for (uint32_t i = 0; i < 8; ++i) { eighth_[i] = root(8, i); }
  }
  // k < n
  HostC at(uint32_t k) const {
    if (k % n8_ == 0) { return eighth_[k / n8_]; }  // zeros and equal parts exactly
    const auto &a = lo_[k & ((1u << sh_) - 1)], &b = hi_[k >> sh_];
    return HostC{(double)(a.first * b.first - a.second * b.second), -(double)(a.first * b.second + a.second * b.first)};
  }
  uint32_t lo_shift() const { return (uint32_t)sh_; }
  std::vector<HostC> lo() const { return rounded(lo_); }  // w_n^i
  std::vector<HostC> hi() const { return rounded(hi_); }  // w_n^(i << lo_shift())

 private:
  using Table = std::vector<std::pair<long double, long double>>;  // cos, sin
  static std::vector<HostC> rounded(const Table& t) {
    std::vector<HostC> r;
    r.reserve(t.size());
    for (const auto& x : t) { r.push_back({(double)x.first, (double)-x.second}); }
    return r;
  }
  uint32_t n8_;
  int sh_ = 0;
  Table lo_, hi_;
  HostC eighth_[8];
};

inline bool is_pow2(uint32_t x) { return x && !(x & (x - 1)); }
inline uint32_t log2u(uint32_t x) {
  uint32_t r = 0;
  while ((1u << r) < x) { ++r; }
  return r;
}

// the stage twiddle tables of a length-n line FFT in the tw_offsets(n, rl) layout; thread_order: the
// radix-rl stage's table of a transform with warp-local exchanges, entry k for k = wl_col(thread)
inline std::vector<HostC> stage_tables(uint32_t n, uint32_t rl, uint32_t r1f = 0, uint32_t vmax = 16,
                                       bool thread_order = false) {
  const TwOffsets o = tw_offsets((int)n, (int)rl, (int)r1f, (int)vmax);
  const uint32_t r1 = plan_r1(n, rl, r1f, vmax), m1 = plan_m1(n, rl, r1f, vmax), m2 = plan_m2(n, rl, r1f, vmax);
  std::vector<HostC> t(o.total);
  auto fill = [&](int off, uint32_t R, uint32_t NS, bool perm = false) {
    for (uint32_t r = 0; r < R; ++r) {
      for (uint32_t k = 0; k < NS; ++k) {
        const uint32_t kk = perm ? (uint32_t)wl_col((int)n, (int)rl, (int)vmax, (int)k) : k;
        t[off + r * NS + k] = root((uint64_t)R * NS, (uint64_t)r * kk);
      }
    }
  };
  if (m1 > 1) { fill(o.aM1, m1, r1); }
  if (m2 > 1) { fill(o.aM2, m2, r1 * m1); }
  fill(o.aRL, rl, n / rl, thread_order);
  if (m2 > 1) { fill(o.bM2, m2, rl); }
  if (m1 > 1) { fill(o.bM1, m1, rl * m2); }
  fill(o.bR1, r1, n / r1);
  return t;
}

// the column FFT's stage tables for a column variant (its values a thread V: tw_offsets(H, V/2, 0, V)),
// and after them w_H^k, k = wl_col(t) (k = t without warp-local exchanges), for its threads t < H / (V/2)
inline std::vector<HostC> col_stage_tables(uint32_t H, int variant) {
  const uint32_t v = (uint32_t)col_vpt(variant), rl = v / 2;
  const bool wl = wl_ok((int)H, (int)rl, (int)v);
  std::vector<HostC> r = stage_tables(H, rl, 0, v, wl);
  for (uint32_t t = 0; t < H / rl; ++t) { r.push_back(root(H, wl ? (uint32_t)wl_col((int)H, (int)rl, (int)v, (int)t) : t)); }
  return r;
}

// The column variant a plan of shape W x H starts with (the reference's built-in tune defaults play the same
// part, src/TuneEntry.cpp); owl_plan_set_column_variant overrides it, and gpuowl_b200.tune finds the quickest.
// Measured on B200 with the present kernels, us per squaring alone / three plans in turn / four plans grouped:
//   128 x 256: 8 values a thread 8.6-8.9 / 3.4 / 2.5, 16 values 9.6 / 3.5 / 3.3
//   256 x 256: 8 values 10.7 / 4.2 / 3.2, 16 values 11.0 / 4.5 / 3.4
//   1024 x 1024 (and every shape from H = 512 up): 8 values 32.1 / 24.1 / 27.5, 16 values 28.2 / 19.8 / 23.2
//   4096 x 2560: two CTAs per SM 304 / 281 / 294, one 326 / 307 / 315
// Three choices date from earlier kernels and are not the quickest any more: 512 x 512 (8 values 14.2 / 7.5 /
// 7.5, 16 values 12.8 / 6.9 / 7.0), 2048 x 2560 (one CTA 139 / 133 / 141, two 130 / 124 / 130, but a product
// 314 against 318 three in turn) and the shapes of H <= 128 (8 values 1-5 % quicker).
inline int default_col_variant(uint32_t W, uint32_t H) {
  if ((W == 128 && H == 256) || (W == 256 && H == 256) || (W == 512 && H == 512)) { return COL_V8; }
  if (W == 4096 && H == 2560) { return COL_V16_OCC2; }
  return COL_V16;
}

// Whether the line pass pairs its lanes (kPairMinW of the kernels); its inverse transform's first middle
// stage then reads the half-way row r = M1/2 with the factor that the mirrored butterflies leave on the
// upper half of their sub-transform, conj(w_2R1^k) for w_2R1^k (and the twist's entry for the same row).
inline bool line_pairs(uint32_t W) { return W >= 512; }

// the entries of a line group's record (LineTw) that lines of W points read, and their exponents: entry
// `at` of line x is w_hN^(m x)
struct LineEntry {
  int at;
  uint32_t m;
};
inline std::vector<LineEntry> line_entries(uint32_t W, uint32_t H) {
  const uint32_t hN = W * H, rl = 8, r1 = plan_r1(W, rl), m1 = plan_m1(W, rl), m2 = plan_m2(W, rl);
  const uint32_t S = W / r1, d1 = S / m1, d2 = d1 / m2;
  const bool pairs = line_pairs(W);
  std::vector<LineEntry> v;
  auto put = [&](int at, uint32_t m) { v.push_back({at, m % hN}); };
  for (uint32_t r = 0; r < r1; ++r) { put((int)r, r * S); }
  // d^(2^i) for the table rows 2^i < R that a stage of radix R reads
  for (int i = 0; (2u << i) <= m1; ++i) { put(LineTw::M1 + i, pairs && (2u << i) == m1 ? W / 32 * 31 : d1 << i); }
  for (int i = 0; (2u << i) <= m2; ++i) { put(LineTw::M2 + i, d2 << i); }
  for (int i = 0; (2u << i) <= rl; ++i) { put(LineTw::RL + i, 1u << i); }
  for (uint32_t j = 0; j < std::min(S, 16u); ++j) { put(LineTw::LO + (int)j, j); }
  for (uint32_t j = 0; pairs && j <= S / 32; ++j) {
    put(LineTw::HI + (int)j, 16 * j);
    put(LineTw::HIB + (int)j, hN + 16 * j - W);
  }
  return v;
}

// the line pass's tables: the stage tables of W points, then the record of every line group (LineTw; entries
// that lines of this width do not read are 0); wt2 and iwt2: the weights of the words of every line
inline std::vector<HostC> line_tables(uint32_t W, uint32_t H, const Roots& roots, const double* wt2,
                                      const double* iwt2) {
  const uint32_t rl = 8, hN = W * H, len = (uint32_t)LineTw::len((int)W);
  std::vector<HostC> t = stage_tables(W, rl, 0, 16, true);
  const TwOffsets o = tw_offsets((int)W, (int)rl);
  const uint32_t r1 = plan_r1(W, rl), m1 = plan_m1(W, rl);
  if (line_pairs(W)) {
    for (uint32_t k = 0; k < r1; ++k) {
      HostC& w = t[o.aM1 + m1 / 2 * r1 + k];
      w.y = -w.y;
    }
  }
  const size_t at = t.size();
  t.resize(at + (size_t)H * len);
  const std::vector<LineEntry> entries = line_entries(W, H);
  std::vector<uint32_t> k(entries.size(), 0);  // m x mod hN
  for (uint32_t x = 0; x < H; ++x) {
    HostC* e = t.data() + at + (size_t)(x / 2) * (2 * len) + x % 2;
    for (size_t i = 0; i < entries.size(); ++i) {
      e[2 * entries[i].at] = roots.at(k[i]);
      k[i] += entries[i].m;
      if (k[i] >= hN) { k[i] -= hN; }
    }
    e[2 * LineTw::WT] = HostC{wt2[2 * x], wt2[2 * x + 1]};
    e[2 * LineTw::IWT] = HostC{iwt2[2 * x], iwt2[2 * x + 1]};
  }
  return t;
}

// w_n^i, i < n
inline std::vector<HostC> root_table(uint32_t n) {
  std::vector<HostC> r(n);
  for (uint32_t i = 0; i < n; ++i) { r[i] = root(n, i); }
  return r;
}

struct Tables {
  uint32_t E = 0, N = 0, W = 0, H = 0, hN = 0, loShift = 0;
  std::vector<HostC> twW, twH, twLo, twHi;
  std::vector<double> wt1, iwt1;
  std::vector<uint32_t> p1masks;  // (bigmask, wrapmask) per (line group, pass-1 thread)
};

// lines per pass-1 block; the width FFT's cross-line radix is 16 / kLinesPerBlock
constexpr uint32_t kLinesPerBlock = 2;

// Shapes the library supports: W a power of two in [64, 4096]; H a power of two in
// [64, 4096], or 5 * 2^k in {640, 1280, 2560}.
inline bool h_supported(uint32_t H) {
  return (is_pow2(H) && H >= 64 && H <= 4096) || H == 640 || H == 1280 || H == 2560;
}
inline bool shape_supported(uint32_t W, uint32_t H) { return is_pow2(W) && W >= 64 && W <= 4096 && h_supported(H); }

// The default W x H split of an FFT of n words: for 2^lg, W = 2^((lg-1)/2) <= H;
// for 5 * 2^k the supported H that makes the shape closest to square (ties to the larger H).
inline bool shape_for(uint32_t n, uint32_t* W, uint32_t* H) {
  const uint32_t hN = n / 2;
  if (is_pow2(n)) {
    const uint32_t w = 1u << ((log2u(n) - 1) / 2), h = hN / w;
    if (!shape_supported(w, h)) { return false; }
    *W = w;
    *H = h;
    return true;
  }
  bool found = false;
  double best = 0;
  for (uint32_t h : {2560u, 1280u, 640u}) {
    if (hN % h) { continue; }
    const uint32_t w = hN / h;
    if (!shape_supported(w, h)) { continue; }
    const double d = std::fabs(std::log((double)w / h));
    if (!found || d < best - 1e-9) {
      found = true;
      best = d;
      *W = w;
      *H = h;
    }
  }
  return found;
}

// The big-word and wrap bits of every pass-1 thread's words: thread t of line group g holds
// column j1 = wl_col(t) + (W/RL) r (r < RL = 16/R) of lines j2 = g R + ll (ll < R), words e = 0, 1;
// bit (r R + ll) 2 + e. With X = X1[j1] + X2[2 j2 + e], the weight wraps when X >= N and the
// word is big when X mod N < E mod N.
inline std::vector<uint32_t> word_masks(uint32_t E, uint32_t W, uint32_t H, const uint32_t* x1, const uint32_t* x2) {
  constexpr uint32_t R = kLinesPerBlock, RL = 16 / R;
  const uint32_t T = R * W / 16, G = H / R, N = 2 * W * H, em = E % N;
  std::vector<uint32_t> m(2 * (size_t)G * T), xt(W);  // xt: X1 in thread order
  for (uint32_t th = 0; th < T; ++th) {
    const uint32_t c = (uint32_t)wl_col((int)W, (int)RL, 16, (int)th);
    for (uint32_t r = 0; r < RL; ++r) { xt[th * RL + r] = x1[c + (W / RL) * r]; }
  }
  auto groups = [&](uint32_t g0, uint32_t g1) {
    for (uint32_t g = g0; g < g1; ++g) {
      const uint32_t* xl = x2 + 2 * R * g;  // i = 2 ll + e
      for (uint32_t th = 0; th < T; ++th) {
        uint32_t big = 0, wrap = 0;
        for (uint32_t r = RL; r-- > 0;) {  // from the top bit down
          const uint32_t x = xt[th * RL + r];
          for (uint32_t i = 2 * R; i-- > 0;) {
            const uint32_t X = x + xl[i];
            wrap = 2 * wrap + (X >= N);
            big = 2 * big + (X < em) + (X - N < em);  // unsigned: at most one of the two
          }
        }
        m[2 * ((size_t)g * T + th)] = big;
        m[2 * ((size_t)g * T + th) + 1] = wrap;
      }
    }
  };
  // 1.3 ns a word: 27 ms at 20M words on one thread
  const unsigned nt = N < (1u << 20) ? 1u : std::max(1u, std::min(std::thread::hardware_concurrency(), 8u));
  std::vector<std::thread> pool;
  pool.reserve(nt);
  for (unsigned i = 1; i < nt; ++i) {
    const uint32_t g0 = (uint32_t)((uint64_t)G * i / nt), g1 = (uint32_t)((uint64_t)G * (i + 1) / nt);
    try {
      pool.emplace_back(groups, g0, g1);
    } catch (const std::system_error&) {
      groups(g0, g1);
    }
  }
  groups(0, (uint32_t)((uint64_t)G / nt));
  for (auto& x : pool) { x.join(); }
  return m;
}

inline Tables make_tables(uint32_t E, uint32_t W, uint32_t H) {
  if (!shape_supported(W, H)) { throw std::invalid_argument("unsupported W x H shape"); }
  Tables t;
  t.E = E;
  t.W = W;
  t.H = H;
  t.hN = W * H;
  t.N = 2 * W * H;
  const uint32_t N = t.N;
  const Roots roots(t.hN);
  t.loShift = roots.lo_shift();
  t.twH = col_stage_tables(H, COL_V16);
  t.twLo = roots.lo();
  t.twHi = roots.hi();

  const uint64_t step = N - (E % N);
  std::vector<uint32_t> x1(W), x2(2 * H);
  t.wt1.resize(W);
  t.iwt1.resize(W);
  for (uint32_t j1 = 0; j1 < W; ++j1) {
    uint32_t X = (uint32_t)((step * 2 * H * (uint64_t)j1) % N);
    x1[j1] = X;
    // in the line pass's thread order
    constexpr uint32_t RL = 16 / kLinesPerBlock;
    const uint32_t r = j1 / (W / RL), th = (uint32_t)wl_thr((int)W, (int)RL, 16, (int)(j1 % (W / RL)));
    const uint32_t at = 2 * (th + W / RL * (r / 2)) + r % 2;
    t.wt1[at] = (double)exp2l((long double)X / N);
    t.iwt1[at] = (double)exp2l(-(long double)X / N);
  }
  std::vector<double> wt2(2 * H), iwt2(2 * H);
  const long double norm = 1.0L / (4.0L * (long double)t.hN);
  for (uint32_t i = 0; i < 2 * H; ++i) {
    uint32_t X = (uint32_t)((step * (uint64_t)i) % N);
    x2[i] = X;
    wt2[i] = (double)exp2l((long double)X / N);
    iwt2[i] = (double)(exp2l(-(long double)X / N) * norm);
  }
  t.twW = line_tables(W, H, roots, wt2.data(), iwt2.data());
  t.p1masks = word_masks(E, W, H, x1.data(), x2.data());
  return t;
}

}  // namespace owl
