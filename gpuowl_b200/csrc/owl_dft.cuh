// owl_dft.cuh -- FP64 complex arithmetic and small DFTs in registers, plus the
// shared-memory Stockham stage helpers used by the two pass kernels.
//
// Conventions: forward DFT X[k] = sum_n x[n] w^(nk) with w = exp(-2 pi i / n);
// INV selects w = exp(+2 pi i / n) (unnormalised). All small DFTs take and
// return natural order.
#pragma once
#include <cstdint>
#include "owl_compat.cuh"

namespace owl {

typedef double2 C;

__device__ __forceinline__ C mk(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ C cadd(C a, C b) { return mk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ C csub(C a, C b) { return mk(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ C cneg(C a) { return mk(-a.x, -a.y); }
__device__ __forceinline__ C cconj(C a) { return mk(a.x, -a.y); }
__device__ __forceinline__ C cmul(C a, C b) {
  return mk(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ C cmulc(C a, C b) {
  return mk(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
// a + b c in four FMAs
__device__ __forceinline__ C caddmul(C a, C b, C c) {
  return mk(fma(b.x, c.x, fma(-b.y, c.y, a.x)), fma(b.x, c.y, fma(b.y, c.x, a.y)));
}
__device__ __forceinline__ C csq(C a) { return mk(fma(a.x, a.x, -a.y * a.y), 2.0 * a.x * a.y); }
// multiply by i
__device__ __forceinline__ C cmuli(C a) { return mk(-a.y, a.x); }
// multiply by -i
__device__ __forceinline__ C cmulmi(C a) { return mk(a.y, -a.x); }

template <bool INV> __device__ __forceinline__ C cmulw(C a, C w) { return INV ? cmulc(a, w) : cmul(a, w); }

// w4 = -i (forward) / +i (inverse)
template <bool INV> __device__ __forceinline__ C mul_w4(C a) { return INV ? cmuli(a) : cmulmi(a); }

constexpr double kC1 = 0.92387953251128675613;  // cos(pi/8)
constexpr double kS1 = 0.38268343236508977173;  // sin(pi/8)
constexpr double kSQ = 0.70710678118654752440;  // sqrt(1/2)

// a * w16^M, M a compile-time constant in [0, 16)
template <bool INV, int M> __device__ __forceinline__ C mul_w16(C a) {
  constexpr int m = M & 15;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (m == 8) {
    return cneg(a);
  } else if constexpr (m == 4) {
    return mul_w4<INV>(a);
  } else if constexpr (m == 12) {
    return mul_w4<!INV>(a);
  } else if constexpr (m == 2 || m == 6 || m == 10 || m == 14) {
    // (+-1 +- i) sqrt(1/2): forward w16^2 = (1 - i)/sqrt2
    constexpr int q = m / 2;  // 1,3,5,7 -> w8^q
    C b = a;
    if constexpr (q == 3) { b = mul_w4<INV>(a); }
    if constexpr (q == 5) { b = cneg(a); }
    if constexpr (q == 7) { b = mul_w4<!INV>(a); }
    // b * w8^1
    if constexpr (!INV) {
      return mk((b.x + b.y) * kSQ, (b.y - b.x) * kSQ);
    } else {
      return mk((b.x - b.y) * kSQ, (b.x + b.y) * kSQ);
    }
  } else {
    // odd m: full complex multiply by (cos 2pi m/16, -+sin 2pi m/16)
    constexpr int k = m % 4;     // 1 or 3
    constexpr int quad = m / 4;  // rotation by w4^quad
    constexpr double c = (k == 1) ? kC1 : kS1;
    constexpr double s = (k == 1) ? kS1 : kC1;
    C b = a;
    if constexpr (quad == 1) { b = mul_w4<INV>(a); }
    if constexpr (quad == 2) { b = cneg(a); }
    if constexpr (quad == 3) { b = mul_w4<!INV>(a); }
    // forward: (c - i s), inverse: (c + i s)
    if constexpr (!INV) {
      return mk(fma(b.x, c, b.y * s), fma(b.y, c, -b.x * s));
    } else {
      return mk(fma(b.x, c, -b.y * s), fma(b.y, c, b.x * s));
    }
  }
}

// a * w8^r for r known after unrolling
template <bool INV> __device__ __forceinline__ C mul_w8(C a, int r) {
  switch (r & 7) {
    case 0: return a;
    case 1: return mul_w16<INV, 2>(a);
    case 2: return mul_w16<INV, 4>(a);
    case 3: return mul_w16<INV, 6>(a);
    case 4: return mul_w16<INV, 8>(a);
    case 5: return mul_w16<INV, 10>(a);
    case 6: return mul_w16<INV, 12>(a);
    default: return mul_w16<INV, 14>(a);
  }
}

template <bool INV> __device__ __forceinline__ void dft2(C* v) {
  C a = v[0];
  v[0] = cadd(a, v[1]);
  v[1] = csub(a, v[1]);
}

template <bool INV> __device__ __forceinline__ void dft4s(C& x0, C& x1, C& x2, C& x3) {
  C a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), d = mul_w4<INV>(csub(x1, x3));
  x0 = cadd(a, c);
  x2 = csub(a, c);
  x1 = cadd(b, d);
  x3 = csub(b, d);
}

template <bool INV> __device__ __forceinline__ void dft4(C* v) { dft4s<INV>(v[0], v[1], v[2], v[3]); }

// t with w8 a = kSQ t: a factor w8 costs two additions, and the kSQ rides on the FMAs that take the product
template <bool INV> __device__ __forceinline__ C w8_sum(C a) {
  return INV ? mk(a.x - a.y, a.x + a.y) : mk(a.x + a.y, a.y - a.x);
}
// a +- kSQ t
__device__ __forceinline__ C addq(C a, C t) { return mk(fma(kSQ, t.x, a.x), fma(kSQ, t.y, a.y)); }
__device__ __forceinline__ C subq(C a, C t) { return mk(fma(-kSQ, t.x, a.x), fma(-kSQ, t.y, a.y)); }

// 8 = 4 (over n1, stride 2) x 2: 52 FP64 instructions (56 with the factors w8, w8^3 multiplied out)
template <bool INV> __device__ __forceinline__ void dft8(C* v) {
  C y0 = v[0], y2 = v[2], y4 = v[4], y6 = v[6];
  C y1 = v[1], y3 = v[3], y5 = v[5], y7 = v[7];
  dft4s<INV>(y0, y2, y4, y6);  // Y0[k1], k1 = 0..3 in (y0, y2, y4, y6)
  dft4s<INV>(y1, y3, y5, y7);  // Y1[k1]
  const C t3 = w8_sum<INV>(y3), t7 = w8_sum<INV>(mul_w4<INV>(y7));
  y5 = mul_w4<INV>(y5);
  v[0] = cadd(y0, y1);
  v[4] = csub(y0, y1);
  v[1] = addq(y2, t3);
  v[5] = subq(y2, t3);
  v[2] = cadd(y4, y5);
  v[6] = csub(y4, y5);
  v[3] = addq(y6, t7);
  v[7] = subq(y6, t7);
}

// 16 = 4 (over n1, stride 4) x 4: 152 FP64 instructions (160 with the factors w8 multiplied out)
template <bool INV> __device__ __forceinline__ void dft16(C* v) {
  C y[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) { y[i] = v[i]; }
  // step 1: for n2: DFT4 over n1 of x[4 n1 + n2]; result k1 kept at index n2 + 4 k1
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) { dft4s<INV>(y[n2], y[n2 + 4], y[n2 + 8], y[n2 + 12]); }
  // step 2: for k1: DFT4 over n2 of the values times w16^(n2 k1) -> X[k1 + 4 k2]
  {
    C a = y[0], b = y[1], c = y[2], d = y[3];
    dft4s<INV>(a, b, c, d);
    v[0] = a;
    v[4] = b;
    v[8] = c;
    v[12] = d;
  }
#pragma unroll
  for (int k1 = 1; k1 < 4; k1 += 2) {  // the middle factor is w8 or w8^3
    const C a = y[4 * k1], t = w8_sum<INV>(k1 == 1 ? y[4 * k1 + 2] : mul_w4<INV>(y[4 * k1 + 2]));
    const C b = k1 == 1 ? mul_w16<INV, 1>(y[4 * k1 + 1]) : mul_w16<INV, 3>(y[4 * k1 + 1]);
    const C d = k1 == 1 ? mul_w16<INV, 3>(y[4 * k1 + 3]) : mul_w16<INV, 9>(y[4 * k1 + 3]);
    const C p = addq(a, t), m = subq(a, t), e = cadd(b, d), f = mul_w4<INV>(csub(b, d));
    v[k1] = cadd(p, e);
    v[k1 + 8] = csub(p, e);
    v[k1 + 4] = cadd(m, f);
    v[k1 + 12] = csub(m, f);
  }
  {  // k1 = 2: the factors w8, w4, w8^3
    const C a = y[8], c = mul_w4<INV>(y[10]), tb = w8_sum<INV>(y[9]), td = w8_sum<INV>(mul_w4<INV>(y[11]));
    const C p = cadd(a, c), m = csub(a, c), e = cadd(tb, td), f = mul_w4<INV>(csub(tb, td));
    v[2] = addq(p, e);
    v[10] = subq(p, e);
    v[6] = addq(m, f);
    v[14] = subq(m, f);
  }
}

constexpr double kC51 = 0.30901699437494742410;   // cos(2 pi / 5)
constexpr double kC52 = -0.80901699437494742410;  // cos(4 pi / 5)
constexpr double kS51 = 0.95105651629515357212;   // sin(2 pi / 5)
constexpr double kS52 = 0.58778525229247312917;   // sin(4 pi / 5)

// 5-point DFT: with t1 = x1 + x4, t2 = x2 + x3, t3 = x1 - x4, t4 = x2 - x3,
// X1,4 = x0 + c1 t1 + c2 t2 -/+ i (s1 t3 + s2 t4), X2,3 = x0 + c2 t1 + c1 t2 -/+ i (s2 t3 - s1 t4)
// (signs of the i terms flipped for the inverse)
template <bool INV> __device__ __forceinline__ void dft5(C* v) {
  const C x0 = v[0];
  const C t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
  const C t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
  const C a1 = mk(x0.x + kC51 * t1.x + kC52 * t2.x, x0.y + kC51 * t1.y + kC52 * t2.y);
  const C a2 = mk(x0.x + kC52 * t1.x + kC51 * t2.x, x0.y + kC52 * t1.y + kC51 * t2.y);
  const C b1 = mk(kS51 * t3.x + kS52 * t4.x, kS51 * t3.y + kS52 * t4.y);
  const C b2 = mk(kS52 * t3.x - kS51 * t4.x, kS52 * t3.y - kS51 * t4.y);
  const C ib1 = INV ? cmulmi(b1) : cmuli(b1);
  const C ib2 = INV ? cmulmi(b2) : cmuli(b2);
  v[0] = cadd(x0, cadd(t1, t2));
  v[1] = csub(a1, ib1);
  v[4] = cadd(a1, ib1);
  v[2] = csub(a2, ib2);
  v[3] = cadd(a2, ib2);
}

// 20 = 4 x 5, coprime factors: n = 5 n1 + 4 n2, k = 5 k1 + 16 k2 (mod 20), no twiddles between
template <bool INV> __device__ __forceinline__ void dft20(C* v) {
#pragma unroll
  for (int n2 = 0; n2 < 5; ++n2) { dft4s<INV>(v[4 * n2], v[(4 * n2 + 5) % 20], v[(4 * n2 + 10) % 20], v[(4 * n2 + 15) % 20]); }
  C y[20];
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    C z[5];
#pragma unroll
    for (int n2 = 0; n2 < 5; ++n2) { z[n2] = v[(5 * k1 + 4 * n2) % 20]; }
    dft5<INV>(z);
#pragma unroll
    for (int k2 = 0; k2 < 5; ++k2) { y[(5 * k1 + 16 * k2) % 20] = z[k2]; }
  }
#pragma unroll
  for (int k = 0; k < 20; ++k) { v[k] = y[k]; }
}

template <int R, bool INV> __device__ __forceinline__ void dftR(C* v) {
  if constexpr (R == 20) {
    dft20<INV>(v);
  } else if constexpr (R == 5) {
    dft5<INV>(v);
  } else if constexpr (R == 2) {
    dft2<INV>(v);
  } else if constexpr (R == 4) {
    dft4<INV>(v);
  } else if constexpr (R == 8) {
    dft8<INV>(v);
  } else {
    static_assert(R == 16, "radix");
    dft16<INV>(v);
  }
}

// shared-memory index padding: one 16-byte pad per 2^PS elements
template <int PS> __device__ __forceinline__ int pad(int i) { return i + (i >> PS); }

constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x / 2); }

// ---- Stockham stage helpers for one line of N complex values held by N/VPT
// threads, VPT (16 or 8) values per thread. Stage radix R (R divides VPT, or 5):
// thread `tl` runs butterflies j = tl + (N/VPT) b, b < VPT/R, inputs x[j + r N/R],
// twiddle w_(NS R)^(r (j mod NS)), outputs y[(j/NS) NS R + j mod NS + r NS].

// butterflies per thread of a radix-R stage (radix 5 leaves the last one to some threads only)
template <int R, int VPT = 16> constexpr int st_nb() { return (VPT + R - 1) / R; }
template <int R, int N, int VPT = 16> __device__ __forceinline__ bool st_has(int j) {
  return (VPT % R == 0) || j < N / R;
}
// j mod NS and j / NS for j >= 0 (mask and shift when NS is a power of two)
template <int NS> __device__ __forceinline__ int smod(int j) {
  if constexpr ((NS & (NS - 1)) == 0) { return j & (NS - 1); } else { return (int)((unsigned)j % (unsigned)NS); }
}
template <int NS> __device__ __forceinline__ int sdiv(int j) { return (int)((unsigned)j / (unsigned)NS); }

template <int R, int N, int PS, int VPT = 16> __device__ __forceinline__ void st_load(const C* buf, int tl, C* v) {
#pragma unroll
  for (int b = 0; b < st_nb<R, VPT>(); ++b) {
    int j = tl + (N / VPT) * b;
    if (!st_has<R, N, VPT>(j)) { continue; }
#pragma unroll
    for (int r = 0; r < R; ++r) { v[b * R + r] = buf[pad<PS>(j + r * (N / R))]; }
  }
}

// Stage twiddles. tab is the stage's [r][k] table, entry r * NS + k = w_(R NS)^(r k); the rows r = 1, 2, 3,
// 4, 8, 12 are read (each correctly rounded) and the other powers are products of two of them, which
// keeps the L1 data path free for the exchanges (all rows read: 101.4 us per iteration at 8M, these 100.4).
//
// Twist: the inter-pass twiddle w_hN^(x y) of line x, y the index along it, rides on the stage twiddles
// of the transform that reads it: a stage of radix R at product NS has the step w_(NS R)^k d with
// d = w_hN^(x N/(NS R)) instead of w_(NS R)^k, so that the multiplication of every point (8 FP64
// instructions a point for generating and applying it) becomes one product per table value and, in the
// first stage, one multiplication. d[e * ds] for e = 0 .. 3 is d, d^2, d^4, d^8 (read if TWIST).
template <bool INV> __device__ __forceinline__ void twmul(C& v, C w) { v = cmulw<INV>(v, w); }
template <int R, bool TWIST>
__device__ __forceinline__ C tw_row(const C* __restrict__ tab, int ns, int k, int e, const C* d, int ds) {
  C w = __ldg(tab + (1 << e) * ns + k);
  if constexpr (TWIST) { w = cmul(w, d[e * ds]); }
  return w;
}
template <int R, bool INV, bool TWIST>
__device__ __forceinline__ void tw_mul(C* x, const C* __restrict__ tab, int ns, int k, const C* d = nullptr, int ds = 1) {
  const C w1 = tw_row<R, TWIST>(tab, ns, k, 0, d, ds);
  twmul<INV>(x[1], w1);
  if constexpr (R > 2) {
    const C w2 = tw_row<R, TWIST>(tab, ns, k, 1, d, ds);
    const C w3 = TWIST ? cmul(w1, w2) : __ldg(tab + 3 * ns + k);
    twmul<INV>(x[2], w2);
    twmul<INV>(x[3], w3);
    if constexpr (R > 4) {
      const C w4 = tw_row<R, TWIST>(tab, ns, k, 2, d, ds);
      twmul<INV>(x[4], w4);
      if constexpr (R > 5) {
        twmul<INV>(x[5], cmul(w4, w1));
        twmul<INV>(x[6], cmul(w4, w2));
        twmul<INV>(x[7], cmul(w4, w3));
      }
      if constexpr (R >= 16) {
        const C w8 = tw_row<R, TWIST>(tab, ns, k, 3, d, ds);
        const C w12 = TWIST ? cmul(w8, w4) : __ldg(tab + 12 * ns + k);
        twmul<INV>(x[8], w8);
        twmul<INV>(x[9], cmul(w8, w1));
        twmul<INV>(x[10], cmul(w8, w2));
        twmul<INV>(x[11], cmul(w8, w3));
        twmul<INV>(x[12], w12);
        twmul<INV>(x[13], cmul(w12, w1));
        twmul<INV>(x[14], cmul(w12, w2));
        twmul<INV>(x[15], cmul(w12, w3));
        if constexpr (R == 20) {
          const C w16 = __ldg(tab + 16 * ns + k);
          twmul<INV>(x[16], w16);
          twmul<INV>(x[17], cmul(w16, w1));
          twmul<INV>(x[18], cmul(w16, w2));
          twmul<INV>(x[19], cmul(w16, w3));
        }
      }
    }
  }
}

// the stage twiddles times base (radix 8 and 16; forward)
template <int R> __device__ __forceinline__ void tw_mul_base(C* x, const C* __restrict__ tab, int ns, int k, C base) {
  static_assert(R == 8 || R == 16, "radix");
  const C w1 = __ldg(tab + ns + k), w2 = __ldg(tab + 2 * ns + k), w4 = __ldg(tab + 4 * ns + k);
  const C lo[4] = {w1, w1, w2, __ldg(tab + 3 * ns + k)};
  C hi[4] = {base, cmul(base, w4), base, base};
  if constexpr (R == 16) {
    const C w8 = __ldg(tab + 8 * ns + k);
    hi[2] = cmul(base, w8);
    hi[3] = cmul(base, __ldg(tab + 12 * ns + k));
  }
#pragma unroll
  for (int r = 0; r < R; ++r) { x[r] = cmul(x[r], (r & 3) == 0 ? hi[r >> 2] : cmul(hi[r >> 2], lo[r & 3])); }
}

// radix-R butterfly of inputs that carry the stage twiddles
template <int R, bool INV, bool TWIST>
__device__ __forceinline__ void tw_dft(C* x, const C* __restrict__ tab, int ns, int k, const C* d, int ds = 1) {
  static_assert(!TWIST || R != 5, "twisted radix");
  tw_mul<R, INV, TWIST>(x, tab, ns, k, d, ds);
  dftR<R, INV>(x);
}

// twiddles and DFTs of a Stockham stage (NS > 1)
template <int R, int N, int NS, bool INV, int VPT = 16>
__device__ __forceinline__ void st_tdft(int tl, C* v, const C* __restrict__ tab) {
#pragma unroll
  for (int b = 0; b < st_nb<R, VPT>(); ++b) {
    int j = tl + (N / VPT) * b;
    if (!st_has<R, N, VPT>(j)) { continue; }
    tw_dft<R, INV, false>(v + b * R, tab, NS, smod<NS>(j), nullptr);
  }
}

template <int R, bool INV, int VPT = 16> __device__ __forceinline__ void st_dft(C* v) {
#pragma unroll
  for (int b = 0; b < st_nb<R, VPT>(); ++b) { dftR<R, INV>(v + b * R); }
}

template <int R, int N, int NS, int PS, int VPT = 16> __device__ __forceinline__ void st_store(C* buf, int tl, const C* v) {
#pragma unroll
  for (int b = 0; b < st_nb<R, VPT>(); ++b) {
    int j = tl + (N / VPT) * b;
    if (!st_has<R, N, VPT>(j)) { continue; }
    int base = sdiv<NS>(j) * NS * R + smod<NS>(j);
#pragma unroll
    for (int r = 0; r < R; ++r) { buf[pad<PS>(base + r * NS)] = v[b * R + r]; }
  }
}

// Radix plan for a line of N points whose last inverse / first forward stage
// (radix RL) is split across lines or columns: N = R1 * M1 * M2 * RL.
// "A order" runs the stages R1, M1, M2, RL; "B order" runs RL, M2, M1, R1.
// n = 2^a or 5 * 2^a; the factor 5 is the M2 stage or part of a first radix of 20. r1f != 0 forces the
// first radix (the split-precision column pass runs a 32-point first stage).
// vmax: the largest radix (the values per thread). 2560 and 1280 points at 16 values a thread start with
// radix 20, run by 4 of every 5 threads: one stage and exchange less than 16 x 4 x 5 x 8, and 20
// sub-transforms that divide among the CTA's 10 or 5 warps (20M: column pass 169 -> 114 us; 5M: 33 -> 24).
__host__ __device__ constexpr int plan_r1(int n, int rl, int r1f = 0, int vmax = 16) {
  return r1f ? r1f : ((n == 2560 || n == 1280) && rl == 8 && vmax == 16 ? 20 : (n / rl >= vmax ? vmax : n / rl));
}
__host__ __device__ constexpr int plan_rest2(int n, int rl, int r1f = 0, int vmax = 16) { return n / rl / plan_r1(n, rl, r1f, vmax); }
__host__ __device__ constexpr int plan_m1(int n, int rl, int r1f = 0, int vmax = 16) {
  return plan_rest2(n, rl, r1f, vmax) % 5 == 0
             ? plan_rest2(n, rl, r1f, vmax) / 5
             : (plan_rest2(n, rl, r1f, vmax) >= vmax ? vmax : plan_rest2(n, rl, r1f, vmax));
}
__host__ __device__ constexpr int plan_m2(int n, int rl, int r1f = 0, int vmax = 16) {
  return plan_rest2(n, rl, r1f, vmax) / plan_m1(n, rl, r1f, vmax);
}

// Column-pass tile variants, chosen per plan (owl_plan_set_column_variant; gpuowl_b200.tune times
// them per shape): the values a thread holds (which fixes the radix plan and the threads of a CTA)
// and the CTAs per SM that the launch bounds ask for.
//   COL_V16       16 values a thread, H/8 threads a CTA: every H
//   COL_V8         8 values a thread, H/4 threads (twice the threads at half the registers; the radix
//                  plan 8 x ... x 4): H a power of two up to 2048, 640 and 1280
//   COL_V16_OCC2  16 values a thread at two CTAs per SM (102 registers, a few spilled): H = 2560,
//                  whose default runs one 320-thread CTA of 168 registers per SM
// COL_AUTO (0) stands for the shape's default (owl_tables.hpp: default_col_variant).
enum : int { COL_AUTO = 0, COL_V16 = 1, COL_V8 = 2, COL_V16_OCC2 = 3 };
__host__ __device__ constexpr bool col_variant_ok(int H, int v) {
  return v == COL_V16 || (v == COL_V8 && ((((H & (H - 1)) == 0) && H <= 2048) || H == 640 || H == 1280)) ||
         (v == COL_V16_OCC2 && H == 2560);
}
__host__ __device__ constexpr int col_vpt(int v) { return v == COL_V8 ? 8 : 16; }
// the CTAs per SM of the column pass's launch bounds (0: the kernel's own rule)
__host__ __device__ constexpr int col_minb(int v) { return v == COL_V16_OCC2 ? 2 : 0; }

// CTAs per SM that the pass kernels' launch bounds ask for: enough for 16 resident warps at most
// 128 registers a thread (T threads a CTA; at most 32 CTAs an SM). Without the hint the kernels of
// the small FFTs (32- to 128-thread CTAs) took 200-255 registers, which left 8-10 warps on an SM.
constexpr int occ_blocks(int T) {
  return T >= 512 ? 1 : (16 / ((T + 31) / 32) > 32 ? 32 : 16 / ((T + 31) / 32));
}

// Stage twiddle tables, one per stage with twiddles, each laid out [r][k]:
// entry r * NS + k = w_(R NS)^(r k) (forward sign), so that a warp's threads
// (consecutive k) read one contiguous run per r. Offsets in complex elements.
struct TwOffsets {
  int aM1, aM2, aRL, bM2, bM1, bR1, total;
};
constexpr TwOffsets tw_offsets(int n, int rl, int r1f = 0, int vmax = 16) {
  const int r1 = plan_r1(n, rl, r1f, vmax), m1 = plan_m1(n, rl, r1f, vmax), m2 = plan_m2(n, rl, r1f, vmax);
  TwOffsets o{};
  o.aM1 = 0;
  o.aM2 = o.aM1 + (m1 > 1 ? m1 * r1 : 0);
  o.aRL = o.aM2 + (m2 > 1 ? m2 * r1 * m1 : 0);
  o.bM2 = o.aRL + n;
  o.bM1 = o.bM2 + (m2 > 1 ? m2 * rl : 0);
  o.bR1 = o.bM1 + (m1 > 1 ? m1 * rl * m2 : 0);
  o.total = o.bR1 + n;
  return o;
}

// Whether a pair of n-point rows runs its middle exchanges inside warps (Wl): its first radix hands every
// warp whole sub-transforms and leaves a power of two. False for 640 points and for 1280 at 8 values a
// thread (a factor 5 stays in the middle stages) and for 2048 points at 8 values a thread (8
// sub-transforms, 16 warps).
__host__ __device__ constexpr bool wl_ok(int n, int rl, int vmax) {
  return plan_rest2(n, rl, 0, vmax) % 5 != 0 && (2 * n / vmax <= 32 || plan_r1(n, rl, 0, vmax) % (2 * n / vmax / 32) == 0);
}
// the column t' of thread t in a Wl transform's radix-RL stage, and back
__host__ __device__ constexpr int wl_col(int n, int rl, int vmax, int t) {
  const int r1 = plan_r1(n, rl, 0, vmax), m = n / rl / r1;
  return t / m + r1 * (t % m);
}
__host__ __device__ constexpr int wl_thr(int n, int rl, int vmax, int c) {
  const int r1 = plan_r1(n, rl, 0, vmax), m = n / rl / r1;
  return (c % r1) * m + c / r1;
}

template <int N, int RL, int R1F = 0, int VPT = 16> struct Plan {
  static constexpr int RLAST = RL;
  static constexpr int R1 = plan_r1(N, RL, R1F, VPT);
  static constexpr int M1 = plan_m1(N, RL, R1F, VPT);
  static constexpr int M2 = plan_m2(N, RL, R1F, VPT);
  static constexpr TwOffsets TW = tw_offsets(N, RL, R1F, VPT);
  static_assert(R1 * M1 * M2 * RL == N, "plan");
  static_assert(M2 >= 1 && M2 <= VPT, "plan depth");
  static_assert(M1 <= VPT && (VPT % M1 == 0), "plan: first middle radix must divide the values per thread");
  static_assert(M2 == 5 || (VPT % M2 == 0), "plan: second middle radix 5 or a divisor of the values per thread");
  static_assert(R1 >= 4, "first radix too small for conflict-free padding");
};

// What the line pass needs to know of a group of two lines x = 2 g, 2 g + 1, one contiguous record that
// the CTA copies to shared memory while its state loads are under way (entry i of line x at 2 i + x % 2):
// the first stage's steps w_hN^(x r W/R1), r < 16; the twists d, d^2, d^4, d^8 of the stages M1 and M2
// and d, d^2, d^4 of the radix-RL stage; w_hN^(x j) as LO[j % 16] HI[j / 16], or for the second of paired
// lanes w_hN^(x (j - W)) as LO[j % 16] HIB[j / 16]; the lines' weights (wt2 and iwt2 of words e = 0, 1).
// Read one by one where they are used, every one of these was an L2 round trip of its own per CTA, and
// the two-level w_hN table two gathers of up to 32 wavefronts.
struct LineTw {
  static constexpr int M1 = 16, RL = 20, WT = 23, IWT = 24, LO = 25, HI = 41, HIB = 50, M2 = 59;
  // length of the record of lines of w points (up to 256 points: no HI, S = W/R1 <= 16 entries of LO)
  __host__ __device__ static constexpr int len(int w) {
    return w <= 256 ? LO + (w == 256 ? 16 : 8) : (w <= 2048 ? M2 : M2 + 4);
  }
};

// ---- The transform of two rows (lines or columns) whose middle exchanges stay inside a warp ----
//
// A CTA of T = 2 N / VPT threads holds two rows of N = R1 M1 M2 RL points. The first (A order) or
// last (B order) radix-R1 stage leaves R1 independent sub-transforms of S = N / R1 points per row,
// sub-transform q in the shared-memory region (row, q); a warp then owns the regions of NSUB = R1 /
// warps values of q in both rows and runs the remaining stages in them with no barrier but its own.
// One exchange of the transform is left that needs the whole CTA. A column pass has 2 block barriers, one
// for each direction, and a fused line pass 4 (two more for its ticket and its record), where two barriers
// per exchange made 9 to 11: at 8M barriers were the line pass's top stall.
//
// Index maps, A order (input index i = j + S r, output index n = q + R1 (p + M n2), M = M1 M2,
// p = p1 + M1 p2; B order is the same graph backwards):
//   region (row, q) starts at row RS + q SQ; after the first stage it holds j at j;
//   after stage M1 it holds (p, jl) at p (RL + 1) + jl (M2 = 1) or (p1, j') at p1 RL M2 + j';
//   after stage M2 it holds (p, jl) at p (RL + 1) + jl;
//   the radix-RL stage runs (q, p) of both rows in thread t = q M + p, whose outputs are n = t' + R1 M n2
//   with t' = wl_col(t) = q + R1 p. Tables that this stage reads are stored in thread order.
// Every access is free of bank conflicts: 8 neighbouring lanes read or write 8 neighbouring elements,
// elements RL + 1 apart, or 4 neighbours in each row with RS = 4 mod 8.
template <int N, int RL, int VPT = 16> struct Wl {
  using P = Plan<N, RL, 0, VPT>;
  static constexpr int R1 = P::R1, M1 = P::M1, M2 = P::M2, M = M1 * M2, S = N / P::R1;
  static constexpr int T = 2 * N / VPT;
  static constexpr int NW = T > 32 ? T / 32 : 1;
  static constexpr int LANES = T > 32 ? 32 : T;
  static constexpr bool ok = wl_ok(N, RL, VPT);
  static constexpr int NSUB = R1 / NW;
  static constexpr int SQ = M * (RL + 1);
  static constexpr int RS = N + N / RL + 4;
};
// barrier of a warp (its first T threads in a CTA of T < 32)
template <int T> __device__ __forceinline__ void wl_sync() { warp_sync(T >= 32 ? 0xffffffffu : ((1u << (T & 31)) - 1u)); }

// row and q of butterfly group gq (2 NSUB groups a warp); MIRROR: row 1 runs R1 - 1 - q
template <typename G, bool MIRROR> __device__ __forceinline__ void wl_group(int warp, int gq, int& row, int& q) {
  // RL = 8: q fastest, RL = 4: the row fastest, so that 8 neighbouring lanes never meet in a bank
  const int ql = (G::P::RLAST == 4) ? gq / 2 : gq % G::NSUB;
  row = (G::P::RLAST == 4) ? gq % 2 : gq / G::NSUB;
  q = warp * G::NSUB + ql;
  if (MIRROR && row == 1) { q = G::R1 - 1 - q; }
}

// One middle stage of a warp: radix R; ld / st give the element of (butterfly u, input or output r) inside
// a region, kf the twiddle index; with TWIST d + row is the row's twist, entries two apart (LineTw).
template <typename G, bool MIRROR, int R, bool INV, bool TWIST, int VPT, typename LD, typename ST, typename KF>
__device__ __forceinline__ void wl_stage(C* smem, int t, const C* __restrict__ tab, int ns,
                                         const C* d, LD ld, ST st, KF kf) {
  constexpr int U = G::S / R;  // butterflies of a region
  constexpr int NB = VPT / R;
  const int warp = t / 32, lane = t % 32;
  C u[VPT];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int f = lane + G::LANES * b;
    int row, q;
    wl_group<G, MIRROR>(warp, f / U, row, q);
    const C* reg = smem + row * G::RS + q * G::SQ;
#pragma unroll
    for (int r = 0; r < R; ++r) { u[b * R + r] = reg[ld(f % U, r)]; }
  }
  wl_sync<G::T>();
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int f = lane + G::LANES * b;
    int row, q;
    wl_group<G, MIRROR>(warp, f / U, row, q);
    tw_dft<R, INV, TWIST>(u + b * R, tab, ns, kf(f % U, q), d + row, 2);
    C* reg = smem + row * G::RS + q * G::SQ;
#pragma unroll
    for (int r = 0; r < R; ++r) { reg[st(f % U, r)] = u[b * R + r]; }
  }
  wl_sync<G::T>();
}

// the middle stages in A order (after the first stage's block exchange, before the radix-RL stage);
// TWIST: d is the line group's record (LineTw). GAP: the upper half of every region after the block
// exchange starts GAP elements late (the line pass's paired lanes)
template <int N, int RL, int VPT, bool MIRROR, bool INV, bool TWIST, int GAP = 0>
__device__ __forceinline__ void wl_middle_a(C* smem, int t, const C* __restrict__ tw, const C* d) {
  using G = Wl<N, RL, VPT>;
  using P = typename G::P;
  static_assert(GAP == 0 || G::M1 > 1, "the gap lies before a middle stage");
  if constexpr (G::M1 > 1) {
    constexpr int U = G::S / G::M1;  // = RL M2
    wl_stage<G, MIRROR, G::M1, INV, TWIST, VPT>(
        smem, t, tw + P::TW.aM1, G::R1, d + 2 * LineTw::M1,
        [](int u, int r) { return u + U * r + (2 * r >= G::M1 ? GAP : 0); },
        [](int u, int r) { return G::M2 == 1 ? r * (RL + 1) + u : r * U + u; }, [](int, int q) { return q; });
  }
  if constexpr (G::M2 > 1) {
    wl_stage<G, MIRROR, G::M2, INV, TWIST, VPT>(
        smem, t, tw + P::TW.aM2, G::R1 * G::M1, d + 2 * LineTw::M2,
        [](int u, int r) { return (u / RL) * (RL * G::M2) + u % RL + RL * r; },
        [](int u, int r) { return (u / RL + G::M1 * r) * (RL + 1) + u % RL; },
        [](int u, int q) { return q + G::R1 * (u / RL); });
  }
}
// the middle stages in B order (after the radix-RL stage, before the last stage's block exchange)
template <int N, int RL, int VPT, bool MIRROR, bool INV, int GAP = 0>
__device__ __forceinline__ void wl_middle_b(C* smem, int t, const C* __restrict__ tw) {
  using G = Wl<N, RL, VPT>;
  using P = typename G::P;
  static_assert(GAP == 0 || G::M1 > 1, "the gap lies after a middle stage");
  if constexpr (G::M2 > 1) {
    wl_stage<G, MIRROR, G::M2, INV, false, VPT>(
        smem, t, tw + P::TW.bM2, RL, nullptr,
        [](int u, int r) { return (u / RL + G::M1 * r) * (RL + 1) + u % RL; },
        [](int u, int r) { return (u / RL) * (RL * G::M2) + u % RL + RL * r; }, [](int u, int) { return u % RL; });
  }
  if constexpr (G::M1 > 1) {
    constexpr int U = G::S / G::M1;
    wl_stage<G, MIRROR, G::M1, INV, false, VPT>(
        smem, t, tw + P::TW.bM1, U, nullptr,
        [](int u, int r) { return G::M2 == 1 ? r * (RL + 1) + u : r * U + u; },
        [](int u, int r) { return u + U * r + (2 * r >= G::M1 ? GAP : 0); }, [](int u, int) { return u; });
  }
}
// the region element where thread t's radix-RL inputs (A order) or outputs (B order) of a row start
template <typename G, bool MIRROR> __device__ __forceinline__ int wl_last(int t, int row) {
  int q = t / G::M, p = t % G::M;
  if (MIRROR && row == 1) {
    q = G::R1 - 1 - q;
    p = G::M - 1 - p;
  }
  return row * G::RS + q * G::SQ + p * (G::P::RLAST + 1);
}

}  // namespace owl
