// lbm_fixed.cuh -- the FP64 collisions in 64-bit fixed point on the integer
// pipes.
//
// GB300 issues two FP64 instructions per clock and SM (measured: DFMA, DADD
// and both 64-bit conversions 1.97 each), against about 52 64-bit integer
// additions and 6 products of 64 x 64 -> 64 top bits.  An FP64 step kernel is
// therefore bound by its FP64 instructions (288 per D3Q19 MRT forward cell:
// 144 clocks, while its 312 bytes take 15 at the copy bandwidth).  The
// populations of a flow near rest are numbers of one known size, f_q = w_q +
// a small deviation, so their collision needs no exponents: it runs on
// two's-complement integers x 2^61, whose unit (4e-19) lies below the last
// place of every population it accepts (1.7e-18 for f_q in [1/128, 1/64)).
// Sums are exact, products err by about one unit, and mass and momentum are
// conserved exactly up to the rounding of the results to FP64; the FP64
// expressions round at the size of rho in every sum.
//
// Cells whose populations leave the accepted range (see Window: far from
// equilibrium, negative, not finite) take the FP64 operators of
// lbm_device.cuh, cell by cell, as do models whose constants do not fit
// (FixedModel::ok).
//
// Measured on one GB300 with the objective, over flows and adjoints that fill
// the lattice, FP64 -> fixed point: 256x128x128 D3Q19 MRT step 1.916 -> 0.309 ms
// forward (4.2 TB/s, 0.63 of the copy bandwidth; 0.289 without the objective)
// and 3.081 -> 0.569 ms reverse; 4096x2048 D2Q9 BGK 1.457 -> 0.238 ms (5.4 TB/s,
// 0.80) and 2.907 -> 0.408 ms; 2048x1024 D2Q9 MRT 0.561 -> 0.064 ms and 1.243 ->
// 0.110 ms; 128x64 BGK 5.6 -> 4.2 us and 11.1 -> 6.3 us.  Where no adjoint has
// arrived the reverse step only reads it (256x128x128 0.419 ms in the first 30
// steps).  What bounds them is the FP64 pipe's conversions (54 to 78% busy, two a
// population) beside the integer work, at 15 to 21 of 64 warps per SM; doubles
// built on the integer pipes instead were slower.  Root-mean-square error of
// one collision against extended precision, over the FP64 operators' own:
// 0.14 to 0.40 forward, 0.19 to 0.69 reverse.
#pragma once

#include <type_traits>

#include "lbm_device.cuh"

namespace lbm {
namespace fx {

typedef unsigned long long u64;
typedef unsigned int u32;

// Two's-complement integers of 64 bits whose sums, differences, products and
// shifts wrap.  The collision relies on it: the terms of a bounded result may
// leave the range on the way (a product of a factor above 1/2 does, see mulc), which
// a built-in signed type leaves undefined.
struct i64 {
  u64 v;
  i64() = default;
  template <class T, class = typename std::enable_if<std::is_integral<T>::value>::type>
  __device__ __forceinline__ constexpr i64(T x) : v(static_cast<u64>(x)) {}
  __device__ __forceinline__ explicit operator u64() const { return v; }
  __device__ __forceinline__ explicit operator long long() const { return (long long)v; }
  __device__ __forceinline__ explicit operator int() const { return (int)(u32)v; }
  __device__ __forceinline__ friend i64 operator+(i64 a, i64 b) { return i64(a.v + b.v); }
  __device__ __forceinline__ friend i64 operator-(i64 a, i64 b) { return i64(a.v - b.v); }
  __device__ __forceinline__ friend i64 operator*(i64 a, i64 b) { return i64(a.v * b.v); }
  __device__ __forceinline__ friend i64 operator^(i64 a, i64 b) { return i64(a.v ^ b.v); }
  __device__ __forceinline__ friend i64 operator&(i64 a, i64 b) { return i64(a.v & b.v); }
  __device__ __forceinline__ i64 operator-() const { return i64(0ull - v); }
  __device__ __forceinline__ i64 operator<<(int n) const { return i64(v << n); }
  __device__ __forceinline__ i64 operator>>(int n) const { return i64((long long)v >> n); }
  __device__ __forceinline__ i64& operator+=(i64 b) { return *this = *this + b; }
  __device__ __forceinline__ i64& operator-=(i64 b) { return *this = *this - b; }
  __device__ __forceinline__ bool negative() const { return (long long)v < 0; }
};

constexpr int kScale = 61;   // populations, moments and increments: value * 2^61

// --- words of a double -------------------------------------------------------

__device__ __forceinline__ u32 hi_word(double v) {
#if defined(__CUDA_ARCH__)
  return (u32)__double2hiint(v);
#else
  u64 b;
  memcpy(&b, &v, 8);
  return (u32)(b >> 32);
#endif
}
__device__ __forceinline__ u32 lo_word(double v) {
#if defined(__CUDA_ARCH__)
  return (u32)__double2loint(v);
#else
  u64 b;
  memcpy(&b, &v, 8);
  return (u32)b;
#endif
}
__device__ __forceinline__ double from_words(u32 hi, u32 lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  u64 b = ((u64)hi << 32) | lo;
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}
__device__ __forceinline__ double from_int(i64 v) {
#if defined(__CUDA_ARCH__)
  return __ll2double_rn((long long)v);
#else
  return (double)(long long)v;
#endif
}

// leading zeros of v != 0
__device__ __forceinline__ int clz64(u64 v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return __builtin_clzll(v);
#endif
}

// v * 2^-k to the nearest double (|v| * 2^-k normal or zero).
__device__ __forceinline__ double to_double(i64 v, int k) {
  const double d = from_int(v);
  const u32 h = hi_word(d);
  return from_words(h != 0u ? h - ((u32)k << 20) : 0u, lo_word(d));
}

// --- products ----------------------------------------------------------------

// A product kept apart from the sums it enters.  Without this the compiler
// gathers the subtracted halves of several signed products into one sum and
// drops the carry of its subtraction where the sum's low word is zero: 0 to 7
// of some 4e9 random cells (per model; all of them reverse steps) came out
// wrong by 2^32 units, 4e-8 of a population, and none of 1e10 to 4e10 with it.
// States and adjoints whose words are zero show it at once: without apart,
// 27 of the 36 cases of reverse steps in tests/test_gpu_fixed_words.py fail, over
// all models; with it none does, nor do the sums that have no such product
// (PairDot, the moments).
__device__ __forceinline__ i64 apart(i64 v) {
#if defined(__CUDA_ARCH__)
  asm("" : "+l"(v.v));
#endif
  return v;
}

// The top 64 bits of a * b without the low partial product and the carries of
// the middle ones: short of the exact quotient by less than 3.
__device__ __forceinline__ u64 umul_top(u64 a, u64 b) {
  const u32 ah = (u32)(a >> 32), al = (u32)a, bh = (u32)(b >> 32), bl = (u32)b;
  return (u64)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

constexpr u64 kBias = 1ull << 63;
using u128 = unsigned __int128;

// m * c / 2^64 within two units, c >= 0 and even: (m + 2^63) c / 2^64 - c / 2
// (unsigned products are the cheap ones).  The truncations lose 1.25 on
// average, of which 1 is added back: a quarter too low in the mean.
__device__ __forceinline__ i64 mulc(i64 m, u64 c) {
  return apart((i64)umul_top((u64)m ^ kBias, c) - (i64)(c >> 1) + 1);
}
// A cell's own factor c, with the constant part of mulc prepared: a factor of
// zero (fluid) gives exactly zero, so that nothing is added to the momentum of
// a cell without porosity.
struct Factor {
  u64 c;
  i64 k;
  __device__ __forceinline__ explicit Factor(u64 v) : c(v), k((i64)(v >> 1) - (v != 0ull ? 1 : 0)) {}
  __device__ __forceinline__ i64 times(i64 m) const {
    return apart((i64)umul_top((u64)m ^ kBias, c) - k);
  }
};
// a * b / 2^64 and a * a / 2^64 for signed operands: (a + 2^63)(b + 2^63) =
// a b + 2^63 (a + b) + 2^126.
__device__ __forceinline__ i64 mulr(i64 a, i64 b) {
  return apart((i64)umul_top((u64)a ^ kBias, (u64)b ^ kBias) - ((a >> 1) + (b >> 1)) -
               ((1ll << 62) - 1));
}
__device__ __forceinline__ i64 sqr(i64 a) {
  const u64 u = (u64)a ^ kBias;
  return apart((i64)umul_top(u, u) - a - ((1ll << 62) - 1));
}
// m * c for a signed constant |c| < 2 given as |c| 2^62 and its sign (0, -1).
__device__ __forceinline__ i64 muls(i64 m, u64 c, int neg) {
  const i64 s = (i64)neg, r = (mulc(m, c) << 2) + 1;
  return (r ^ s) - s;
}
// The same, finer, for |m| < 2^58.5.
__device__ __forceinline__ i64 muls_fine(i64 m, u64 c, int neg) {
  const i64 s = (i64)neg, r = (mulc(m << 4, c) + 2) >> 2;
  return (r ^ s) - s;
}

// Accepted range of the populations: each lies within 2^-4 of its share w_q rho
// of the cell's density (velocities up to about 0.17), the rest population in
// [2^-8, 1) (densities up to 2) and the others in [2^-9, 1/2), so that no bit
// of the double falls below 2^-61.  Every moment that the collisions multiply
// is free of the rest equilibrium's part, so it is bounded by the deviations:
// for any combination of accepted populations it stays below 4 (2^63 units);
// sums may wrap on the way.
//
// load(): x = f * 2^61 exactly; ok(): whether the cell is accepted.
struct Window {
  u32 bad = 0u;
  static constexpr u32 kDev = 1u << (kScale - 32 - 4);   // 2^-4 in the high word
  template <int LAT, int q>
  __device__ __forceinline__ i64 load(double f) {
    const u32 h = hi_word(f), l = lo_word(f);
    // f = m 2^(e - 1075) with the 53-bit mantissa m, so x = m << (e - 1014)
    const u32 sh = (h >> 20) - (u32)(1075 - kScale);
    bad |= (q == 0 ? sh - 1u : sh) & ~7u;
    const u32 m = (h & 0xfffffu) | 0x100000u;
#if defined(__CUDA_ARCH__)
    const u32 xh = __funnelshift_l(l, m, sh), xl = __funnelshift_l(0u, l, sh);
#else
    const u64 m64 = (((u64)m << 32) | l) << (sh & 31u);
    const u32 xh = (u32)(m64 >> 32), xl = (u32)m64;
#endif
    return (i64)(((u64)xh << 32) | xl);
  }
  template <int LAT>
  __device__ __forceinline__ bool ok(const i64* x) const {
    using L = Lattice<LAT>;
    u32 rho = 0u, dev = 0u;
    static_for<L::QF>([&](auto Q_) { rho += (u32)((u64)x[decltype(Q_)::value] >> 32); });
    const u32 share = __umulhi(rho, 0x071c71c7u);   // rho / 36
    static_for<L::QF>([&](auto Q_) {
      constexpr int q = decltype(Q_)::value;
      constexpr u32 n = (u32)(36. * L::w(q) + 0.5);
      dev |= (u32)((u64)x[q] >> 32) - (n * share - kDev);
    });
    return (bad | (dev & ~(2u * kDev - 1u))) == 0u;
  }
};

// ---------------------------------------------------------------------------
// D3Q19 MRT + partial bounce-back in population-pair form (mrt3d_pair_collide
// with the equilibrium folded into the rows and the rates into the back-map).
// c[]: s1/63, s2*2/63, s4/12, om/18, s10/36, om/6, s10/12, om/2, s16/4.

enum { C3_E = 0, C3_EPS, C3_Q, C3_PXX, C3_PIXX, C3_PWW, C3_PIWW, C3_P, C3_M };

struct Moments3 {
  i64 s[10], a[10];
  i64 jx, jy, jz;
  i64 r2, r3, r4, r12, r13, r14;   // relaxed odd moments
  __device__ __forceinline__ void pairs(const i64* x) {
    static_for<9>([&](auto D) {
      constexpr int d = decltype(D)::value + 1;
      s[d] = x[d] + x[d + 9];
      a[d] = x[d] - x[d + 9];
    });
  }
  // momentum and the relaxed odd rows
  __device__ __forceinline__ void odd(const FixedModel& m) {
    const i64 ux = a[9] - a[8], vx = a[7] - a[6], X = ux + vx;
    jx = X - a[3];
    const i64 py = a[5] - a[4], qy = a[8] + a[9], Y = py - qy;
    jy = Y - a[2];
    const i64 rz = a[4] + a[5], tz = a[6] + a[7], Z = rz + tz;
    jz = -(Z + a[1]);
    // q + (2/3) j = (5/3)(X + 2 a): the factor is in the constant
    r2 = mulc(X + 2 * a[3], m.c[C3_Q]);
    r3 = mulc(Y + 2 * a[2], m.c[C3_Q]);
    r4 = mulc(2 * a[1] - Z, m.c[C3_Q]);
    r12 = mulc(ux - vx, m.c[C3_M]);
    r13 = mulc(py + qy, m.c[C3_M]);
    r14 = mulc(rz - tz, m.c[C3_M]);
  }
  // Odd part of the back-map of pair d: O_d = -2 sum_odd (M[k][d]/N_k) r_k,
  // a row entry of +-4 counting 4 r (q rows, N = 40) and +-1 counting r.
  template <int d>
  __device__ __forceinline__ i64 O() const {
    i64 v = 0;
    const i64 r[6] = {r2, r3, r4, r12, r13, r14};
    static_for<6>([&](auto K) {
      constexpr int k = decltype(K)::value;
      constexpr int c = mrt3d_m(k < 3 ? k + 2 : k + 9, d);
      if constexpr (c == 1) v -= r[k];
      if constexpr (c == -1) v += r[k];
      if constexpr (c == 4) v -= r[k] << 2;
      if constexpr (c == -4) v += r[k] << 2;
    });
    return v;
  }
};

// f <- PBB(MRT(f)) of one cell whose populations are x (Window::load); im:
// imult.
__device__ __forceinline__ void mrt3d_collide(const i64* x, const Factor& im, const FixedModel& m,
                                              double* f) {
  Moments3 t;
  t.pairs(x);
  const i64* s = t.s;
  const i64* a = t.a;
  t.odd(m);
  // products of the velocity: 2^63 x 2^63 / 2^64 = 2^62 units, halved
  const i64 qx = t.jx << 2, qy = t.jy << 2, qz = t.jz << 2;
  const i64 xx = sqr(qx), yy = sqr(qy), zz = sqr(qz);
  const i64 jsq = (xx + yy + zz) >> 1;
  const i64 t1 = ((xx << 1) - (yy + zz)) >> 1, t2 = (yy - zz) >> 1;
  const i64 sax = (s[1] + s[2]) + s[3];
  const i64 dyz = s[4] + s[5], dxz = s[6] + s[7], dxy = s[8] + s[9];
  const i64 sdg = (dyz + dxz) + dxy;
  // e - e_eq = 19 (sdg - f0 - j^2); (eps - eps_eq)/4 = (9 (f0 - sax) + 2 (sax - sdg))/4
  // - ((we - 3)/4) rho - (wej/4) j^2
  const i64 r0 = mulc((sdg - x[0]) - jsq, m.c[C3_E]);
  const i64 p = x[0] - sax;
  i64 e1 = (p << 1) + (p >> 2) + ((sax - sdg) >> 1) - muls(jsq, m.wej, m.wej_neg);
  if (m.we3) e1 -= muls(x[0] + sax + sdg, m.we3c, m.we3_neg);
  const i64 r1 = mulc(e1, m.c[C3_EPS]);
  const i64 A = (s[3] << 1) - (s[1] + s[2]), B = (dxz + dxy) - (dyz << 1);
  const i64 r5 = mulc(A + B - t1, m.c[C3_PXX]);
  const i64 r6 = mulc(B - (A << 1) - muls(t1, m.wxx, m.wxx_neg), m.c[C3_PIXX]);
  const i64 A2 = s[2] - s[1], B2 = dxy - dxz;
  const i64 r7 = mulc(A2 + B2 - t2, m.c[C3_PWW]);
  const i64 r8 = mulc(B2 - (A2 << 1) - muls(t2, m.wxx, m.wxx_neg), m.c[C3_PIWW]);
  const i64 h9 = mulc(s[8] - s[9] - (mulr(qx, qy) >> 1), m.c[C3_P]);
  const i64 h10 = mulc(s[4] - s[5] - (mulr(qy, qz) >> 1), m.c[C3_P]);
  const i64 h11 = mulc(s[6] - s[7] - (mulr(qx, qz) >> 1), m.c[C3_P]);
  // even back-map: pair sums gain E_d, the rest population d0 (the integers
  // cancel exactly over the cell)
  f[0] = to_double((x[0] + 15 * r0 - 6 * r1) << 1, kScale + 1);
  const i64 cax = 11 * r0 + (r1 << 2), cdg = -(r0 << 3) - r1;
  const i64 P = r5 - (r6 << 1), Q = r5 + r6;
  const i64 R = r7 - (r8 << 1), T = r7 + r8;
  const i64 ax12 = cax + P, c45 = cdg + (Q << 1), cq = cdg - Q;
  const i64 E[10] = {0,        ax12 + R,      ax12 - R,      cax - (P << 1), c45 - h10,
                     c45 + h10, cq + T - h11, cq + T + h11, cq - T - h9,    cq - T + h9};
  static_for<9>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    const i64 sp = s[d] + E[d];
    i64 ap = a[d] + t.template O<d>();
    ap -= im.times(ap << 1);
    // f = (sp +- ap) / 2
    f[d] = to_double(sp + ap, kScale + 1);
    f[d + 9] = to_double(sp - ap, kScale + 1);
  });
}

// ---------------------------------------------------------------------------
// Reverse steps.  The adjoint populations of a cell have no known size but one
// in common: they are brought to integers by the cell's own power of two, so
// that the largest lies in [2^59, 2^60).  The pairs' sums and differences
// enter the transposed collision at a sixteenth of that (|.| < 2^57), which
// leaves its rows room and errs by 2^-57 of the largest, below the rounding
// of an FP64 sum over the cell; the derivative by imult takes the differences
// as they are.

// Whether all of v are finite and below 2^64: the transposed collision at such a state
// takes an adjoint of zero to zero, in FP64 too.
template <int N>
__device__ __forceinline__ bool moderate(const double* v) {
  u32 m = 0u;
  static_for<N>([&](auto Q_) {
    const u32 h = hi_word(v[decltype(Q_)::value]) & 0x7fffffffu;
    m = h > m ? h : m;
  });
  return m < (1087u << 20);
}

template <int BITS>
struct BlockOf {
  int k = 0;       // values * 2^k, the largest below 2^BITS
  int top = 0;     // exponent field of the largest
  bool zero = false, ok = false;
  // scale from the largest magnitude; exponents past these bounds (1e-210,
  // 1e16) and values that are not finite are left to the FP64 operators.
  // zero: no adjoint has arrived at the cell yet, and the transposed
  // collision, which is linear, leaves it so.
  template <int N>
  __device__ __forceinline__ void measure(const double* v) {
    u32 m = 0u;
    static_for<N>([&](auto Q_) {
      const u32 h = hi_word(v[decltype(Q_)::value]) & 0x7fffffffu;
      m = h > m ? h : m;
    });
    top = (int)(m >> 20);
    zero = m == 0u;
    ok = top >= 323 && top <= 1077;
    k = 1022 + BITS - top;
  }
  // no finer than 2^-kmax
  __device__ __forceinline__ void at_most(int kmax) {
    if (zero || k > kmax) {
      k = kmax;
      top = 1022 + BITS - k;
      zero = false;
      ok = true;
    }
  }
  // v * 2^k rounded to the nearest integer.  The conversion runs on the FP64
  // pipe, except that the temperature lattice, whose two scales and FP64 terms
  // keep that pipe busy, builds the integer from the words (512x256 step 11.4
  // -> 10.3 us forward, 24.3 -> 23.4 us reverse; the D3Q19 reverse step, short
  // of registers, went 0.515 -> 0.536 ms with it).
  __device__ __forceinline__ i64 load(double v) const {
#if defined(__CUDA_ARCH__)
    if constexpr (BITS == 60) {
      return __double2ll_rn(from_words(hi_word(v) + ((u32)k << 20), lo_word(v)));
    }
#endif
    const u32 h = hi_word(v);
    const int sh = top - (int)((h >> 20) & 0x7ffu);   // below the largest by 2^sh
    const u64 m = ((u64)((h & 0xfffffu) | 0x100000u) << 32 | lo_word(v)) << (BITS - 52);
    const i64 a = (i64)(((m >> (sh < 63 ? sh : 63)) + 1u) >> 1);
    const i64 s = (i64)((int)h >> 31);
    return (a ^ s) - s;
  }
  // results: 2 lam at the reduced scale
  __device__ __forceinline__ double store(i64 v) const { return to_double(v, k - 3); }
};
using Block = BlockOf<60>;

// -sum a * w over the pairs, a * 2^61 and w in a Block's units (|a| < 0.6, |w|
// < 2^61): products of 31-bit limbs, exact to 2^-86 of the largest.
struct PairDot {
  i64 h = 0, m = 0;   // h 2^62 + m 2^35
  __device__ __forceinline__ void add(i64 a, i64 w) {
    const int ah = (int)(a >> 31), wh = (int)(w >> 31);
    const int al = (int)(a & 0x7fffffff), wl = (int)(w & 0x7fffffff);
    h -= (i64)ah * wh;
    m -= ((i64)ah * wl + (i64)al * wh + (i64)(u64)__umulhi((u32)al << 1, (u32)wl)) >> 4;
  }
  __device__ __forceinline__ double value(const Block& b) const {
    return to_double(h, b.k - 1) + to_double(m, b.k + 26);
  }
};

// one pair: reduced sum and (bounced-back) difference, and its share of the
// derivative by imult, a: the collided difference before partial bounce-back
__device__ __forceinline__ void load_pair(const Block& b, double lam, double lam_opp, i64 a,
                                          const Factor& im, i64& ls, i64& la, PairDot& rev) {
  const i64 u = b.load(lam), v = b.load(lam_opp), w = u - v;
  rev.add(a, w);
  ls = (u + v + 8) >> 4;
  const i64 r = (w + 8) >> 4;
  la = r - im.times(r << 1);
}

// Transpose of mrt3d_collide: lam (adjoint of the output) in, adjoint of the
// input out; returns the sum over the pairs of (collided difference before
// partial bounce-back) * (lam_opp - lam_d), the derivative by imult.  The
// moments keep the forward constants, which makes them twice mrt3d_pair_reverse's.
__device__ __forceinline__ double mrt3d_reverse(const i64* x, double* lam, const Block& b,
                                                const Factor& im, const FixedModel& m) {
  Moments3 t;
  t.pairs(x);
  t.odd(m);
  i64 ls[10], la[10];
  PairDot rev;
  const i64 f0 = (b.load(lam[0]) + 8) >> 4;
  static_for<9>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    load_pair(b, lam[d], lam[d + 9], t.a[d] + t.template O<d>(), im, ls[d], la[d], rev);
  });
  const i64 sax = (ls[1] + ls[2]) + ls[3];
  const i64 dyz = ls[4] + ls[5], dxz = ls[6] + ls[7], dxy = ls[8] + ls[9];
  const i64 sdg = (dyz + dxz) + dxy;
  // the energy row, halved: its weights sum to 96
  const i64 n0 = mulc((sdg << 2) - (15 * f0 + 5 * sax + (sax >> 1)), m.c[C3_E] << 1);
  const i64 u8 = mulc(12 * f0 + sdg - (sax << 2), m.c[C3_EPS]);   // 8 M1, M1 = (s2/252) row
  const i64 A = (ls[3] << 1) - (ls[1] + ls[2]), B = (dxz + dxy) - (dyz << 1);
  const i64 m5 = mulc(A + B, m.c[C3_PXX]), m6 = mulc(B - (A << 1), m.c[C3_PIXX]);
  const i64 A2 = ls[2] - ls[1], B2 = dxy - dxz;
  const i64 m7 = mulc(A2 + B2, m.c[C3_PWW]), m8 = mulc(B2 - (A2 << 1), m.c[C3_PIWW]);
  const i64 m9 = mulc(ls[8] - ls[9], m.c[C3_P]);
  const i64 m10 = mulc(ls[4] - ls[5], m.c[C3_P]);
  const i64 m11 = mulc(ls[6] - ls[7], m.c[C3_P]);
  const i64 ux = la[9] - la[8], vx = la[7] - la[6];
  const i64 py = la[5] - la[4], qy = la[8] + la[9];
  const i64 rz = la[4] + la[5], tz = la[6] + la[7];
  const i64 nx = mulc(ux + vx + (la[3] << 2), m.c[C3_Q]);
  const i64 ny = mulc(py - qy + (la[2] << 2), m.c[C3_Q]);
  const i64 nz = mulc((la[1] << 2) - (rz + tz), m.c[C3_Q]);
  const i64 m12 = mulc(ux - vx, m.c[C3_M]);
  const i64 m13 = mulc(py + qy, m.c[C3_M]);
  const i64 m14 = mulc(rz - tz, m.c[C3_M]);
  // through the quadratic equilibria: half the gradient by j, 2^63 x 2 / 2^64 = 1
  const i64 qx = t.jx << 2, qyv = t.jy << 2, qz = t.jz << 2;
  // 2 n + 2 wej u + 4 (m5 + wxx m6) and alike, u = 2 M1: wej u = (wej/4) u8
  const i64 b0 = (n0 + muls_fine(u8, m.wej, m.wej_neg)) << 1;
  const i64 a56 = m5 + muls_fine(m6, m.wxx, m.wxx_neg), a78 = m7 + muls_fine(m8, m.wxx, m.wxx_neg);
  const i64 gx = mulr(qx, (b0 + (a56 << 2)) << 1) + mulr(qyv, m9 << 1) + mulr(qz, m11 << 1) + 1;
  const i64 gy = mulr(qyv, (b0 + ((a78 - a56) << 1)) << 1) + mulr(qx, m9 << 1) + mulr(qz, m10 << 1) + 1;
  const i64 gz = mulr(qz, (b0 - ((a56 + a78) << 1)) << 1) + mulr(qyv, m10 << 1) + mulr(qx, m11 << 1) + 1;
  // 2 (rR + G): rest n - 18 M1, axes 14 M1, diagonals -n + 4 M1 (we = 3),
  // and 2 (we - 3) M1 in each
  i64 w3 = 0;
  if (m.we3) w3 = muls_fine(u8, m.we3c, m.we3_neg);
  lam[0] = b.store((f0 << 1) + n0 - ((9 * u8 + 2) >> 2) + w3);
  const i64 cax = ((7 * u8 + 2) >> 2) + w3, cdg = ((u8 + 1) >> 1) - n0 + w3;
  const i64 P = m5 - (m6 << 1), Q = m5 + m6;
  const i64 R = m7 - (m8 << 1), T = m7 + m8;
  const i64 ax12 = cax + P, c45 = cdg + (Q << 1), cq = cdg - Q;
  const i64 G_[10] = {0,         ax12 + R,     ax12 - R,     cax - (P << 1), c45 - m10,
                      c45 + m10, cq + T - m11, cq + T + m11, cq - T - m9,    cq - T + m9};
  using L = Lattice<LAT_D3Q19>;
  static_for<9>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    const i64 sp = ls[d] + G_[d];
    // 2 abar: the q rows with the (2/3) j part of their equilibrium (axes
    // 2 e n, diagonals -e n), the m rows, and e . g
    i64 ap = la[d];
    constexpr bool axis = d <= 3;
    if constexpr (L::ex(d) != 0) ap += L::ex(d) * (axis ? gx + (nx << 1) : gx - nx);
    if constexpr (L::ey(d) != 0) ap += L::ey(d) * (axis ? gy + (ny << 1) : gy - ny);
    if constexpr (L::ez(d) != 0) ap += L::ez(d) * (axis ? gz + (nz << 1) : gz - nz);
    if constexpr (mrt3d_m(12, d) != 0) ap -= mrt3d_m(12, d) * m12;
    if constexpr (mrt3d_m(13, d) != 0) ap -= mrt3d_m(13, d) * m13;
    if constexpr (mrt3d_m(14, d) != 0) ap -= mrt3d_m(14, d) * m14;
    lam[d] = b.store(sp + ap);
    lam[d + 9] = b.store(sp - ap);
  });
  return rev.value(b);
}

// ---------------------------------------------------------------------------
// D2Q9 BGK + partial bounce-back in pair form (pairs 1, 3 the diagonals, 2 the
// y and 4 the x axis).  The relaxation is evaluated where it has to be and
// completed by conservation, exactly: the rest population takes what the even
// increments leave of the mass, the axes' odd increments what the diagonals'
// leave of the momentum.
// c[]: om/2, om/6.

enum { C2_HALF_OM = 0, C2_SIXTH_OM };
constexpr u64 kEighteenth = 0x0e38e38e38e38e38ull;   // 2^64 / 18

struct Pairs2 {
  i64 s[5], a[5];
  i64 jx, jy;
  __device__ __forceinline__ explicit Pairs2(const i64* x) {
    static_for<4>([&](auto D) {
      constexpr int d = decltype(D)::value + 1;
      s[d] = x[d] + x[d + 4];
      a[d] = x[d] - x[d + 4];
    });
    jx = (a[1] - a[3]) - a[4];
    jy = -((a[1] + a[3]) + a[2]);
  }
};

// odd increments of the pairs
__device__ __forceinline__ void bgk2_odd(const Pairs2& t, const FixedModel& m, i64* o) {
  o[1] = mulc((t.jx - t.jy) - 6 * t.a[1], m.c[C2_SIXTH_OM]);
  o[3] = mulc(-(t.jx + t.jy) - 6 * t.a[3], m.c[C2_SIXTH_OM]);
  o[4] = o[1] - o[3];
  o[2] = -(o[1] + o[3]);
}

// the collided pairs into populations: f = ((s + E) +- (a + O)(1 - 2 imult)) / 2
__device__ __forceinline__ void finish2(const Pairs2& t, const i64* E, const i64* o,
                                        const Factor& im, double* f) {
  static_for<4>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    const i64 sp = t.s[d] + E[d];
    i64 ap = t.a[d] + o[d];
    ap -= im.times(ap << 1);
    f[d] = to_double(sp + ap, kScale + 1);
    f[d + 4] = to_double(sp - ap, kScale + 1);
  });
}

__device__ __forceinline__ void bgk2_collide(const i64* x, const Factor& im, const FixedModel& m,
                                             double* f) {
  const Pairs2 t(x);
  i64 o[5], E[5];
  bgk2_odd(t, m, o);
  const i64 qx = t.jx << 2, qy = t.jy << 2;
  const i64 xx = sqr(qx), yy = sqr(qy), xy = mulr(qx, qy), sq = xx + yy;   // * 2^62
  const i64 rho = (x[0] + (t.s[1] + t.s[3])) + (t.s[2] + t.s[4]);
  const i64 c = mulc(rho - ((3 * sq) >> 2), kEighteenth);   // (rho - 1.5 j^2) / 18
  // pair sums of the equilibrium: diagonals c + (e.j)^2 / 4, axes 4 c + (e.j)^2
  E[1] = mulc((c + ((sq - (xy << 1)) >> 3) - t.s[1]) << 1, m.c[C2_HALF_OM]);
  E[3] = mulc((c + ((sq + (xy << 1)) >> 3) - t.s[3]) << 1, m.c[C2_HALF_OM]);
  E[2] = mulc(((c << 2) + (yy >> 1) - t.s[2]) << 1, m.c[C2_HALF_OM]);
  E[4] = mulc(((c << 2) + (xx >> 1) - t.s[4]) << 1, m.c[C2_HALF_OM]);
  f[0] = to_double((x[0] - (E[1] + E[2] + E[3] + E[4])) << 1, kScale + 1);
  finish2(t, E, o, im, f);
}

// the end of a reverse step: doubled sums S and differences D of the pairs
__device__ __forceinline__ void store2(const i64* S, const i64* D_, i64 f0, const Block& b,
                                       double* lam) {
  lam[0] = b.store(f0);
  static_for<4>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    lam[d] = b.store(S[d] + D_[d]);
    lam[d + 4] = b.store(S[d] - D_[d]);
  });
}

// pair sums and (bounced-back) differences of the adjoint; the derivative by imult
__device__ __forceinline__ double load2(const double* lam, const Block& b, const Pairs2& t,
                                        const i64* o, const Factor& im, i64* ls, i64* la) {
  PairDot rev;
  static_for<4>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    load_pair(b, lam[d], lam[d + 4], t.a[d] + o[d], im, ls[d], la[d], rev);
  });
  return rev.value(b);
}

// What an objective adds to the adjoint of a 2D cell, in the units of
// Block::store: ev[k] to both populations of pair k (ev[0] to the rest one)
// and +-e_k . (gx, gy) to them.
struct Source2 {
  bool on = false;
  i64 ev[5], gx, gy;
  __device__ __forceinline__ void add(i64* S, i64* F, i64& f0) const {
    if (!on) return;
    f0 += ev[0];
    static_for<4>([&](auto D) {
      constexpr int k = decltype(D)::value + 1;
      S[k] += ev[k];
      F[k] += e_dot<LAT_D2Q9, k>(gx, gy, (i64)0);
    });
  }
};

// Transpose of bgk2_collide: lam + om (E^T lam - lam) with (E^T lam)_i = c0 +
// e_i . c, 36 c0 = 16 lam_0 + (s1 + s3) + 4 (s2 + s4) and 12 c_x = (d1 - d3 -
// 4 d4) + 2 jx (s1 + s3 + 4 s4 - 2 s2 - 8 lam_0) + 3 jy (s3 - s1) (y alike).
__device__ __forceinline__ double bgk2_reverse(const i64* x, double* lam, const Block& b,
                                               const Factor& im, const FixedModel& m,
                                               const Source2& src) {
  const Pairs2 t(x);
  i64 o[5], ls[5], la[5];
  bgk2_odd(t, m, o);
  const i64 v0 = (b.load(lam[0]) + 8) >> 4;
  const double rev = load2(lam, b, t, o, im, ls, la);
  const i64 qx = t.jx << 2, qy = t.jy << 2;
  const i64 D = ls[1] + ls[3], xy = 3 * (ls[3] - ls[1]);
  const i64 c36 = (v0 << 4) + D + ((ls[2] + ls[4]) << 2);
  // 2^63 x 4 / 2^64 = 2
  const i64 cx = (la[1] - la[3] - (la[4] << 2)) +
                 mulr(qx, (D + (ls[4] << 2) - (ls[2] << 1) - (v0 << 3)) << 2) + mulr(qy, xy << 1);
  const i64 cy = -(la[1] + la[3] + (la[2] << 2)) +
                 mulr(qy, (D + (ls[2] << 2) - (ls[4] << 1) - (v0 << 3)) << 2) + mulr(qx, xy << 1);
  const u64 h6 = m.c[C2_SIXTH_OM], h18 = h6 / 3;
  i64 S[5], F[5];
  static_for<4>([&](auto K) {
    constexpr int k = decltype(K)::value + 1;
    using L = Lattice<LAT_D2Q9>;
    S[k] = ls[k] + mulc(c36 - 18 * ls[k], h18);
    i64 ec = -6 * la[k];
    if constexpr (L::ex(k) != 0) ec += L::ex(k) * cx;
    if constexpr (L::ey(k) != 0) ec += L::ey(k) * cy;
    F[k] = la[k] + mulc(ec, h6);
  });
  // 2 (lam_0 + om (c0 - lam_0))
  i64 f0 = (v0 << 1) + mulc(c36 - 36 * v0, h18);
  src.add(S, F, f0);
  store2(S, F, f0, b, lam);
  return rev;
}

// ---------------------------------------------------------------------------
// D2Q9 MRT + partial bounce-back in pair form (IncompressibleMRT2d's moments,
// the equilibria folded into the rows, the rates into the back-map).
// c[]: s1/36, s2/12, s46/6, om/2.

enum { CM_E = 0, CM_EPS, CM_Q, CM_P };

__device__ __forceinline__ void mrt2_odd(const Pairs2& t, const FixedModel& m, i64* o) {
  const i64 r2 = mulc(((t.a[1] - t.a[3]) << 1) + t.a[4], m.c[CM_Q]);
  const i64 r3 = mulc(t.a[2] - ((t.a[1] + t.a[3]) << 1), m.c[CM_Q]);
  o[1] = r3 - r2;
  o[3] = r3 + r2;
  o[4] = -(r2 << 1);
  o[2] = -(r3 << 1);
}

__device__ __forceinline__ void mrt2_collide(const i64* x, const Factor& im, const FixedModel& m,
                                             double* f) {
  const Pairs2 t(x);
  i64 o[5], E[5];
  mrt2_odd(t, m, o);
  const i64 qx = t.jx << 2, qy = t.jy << 2;
  const i64 xx = sqr(qx), yy = sqr(qy), xy = mulr(qx, qy) >> 1;
  const i64 sq = (xx + yy) >> 1;
  const i64 D = t.s[1] + t.s[3], A = t.s[2] + t.s[4];
  // e - e_eq; (eps - eps_eq) / 3
  const i64 r0 = mulc((D << 2) + A - (x[0] << 1) - 3 * sq, m.c[CM_E]);
  const i64 r1 = mulc((x[0] - A) + sq, m.c[CM_EPS]);
  const i64 h4 = mulc((t.s[4] - t.s[2]) - ((xx - yy) >> 1), m.c[CM_P]);
  const i64 h5 = mulc((t.s[3] - t.s[1]) - xy, m.c[CM_P]);
  const i64 dg = -((r0 << 2) + (r1 << 1)), ax = (r0 << 1) + (r1 << 2);
  E[1] = dg + h5;
  E[3] = dg - h5;
  E[2] = ax + h4;
  E[4] = ax - h4;
  f[0] = to_double((x[0] + ((r0 - r1) << 2)) << 1, kScale + 1);
  finish2(t, E, o, im, f);
}

__device__ __forceinline__ double mrt2_reverse(const i64* x, double* lam, const Block& b,
                                               const Factor& im, const FixedModel& m,
                                               const Source2& src) {
  const Pairs2 t(x);
  i64 o[5], ls[5], la[5];
  mrt2_odd(t, m, o);
  const i64 v0 = (b.load(lam[0]) + 8) >> 4;
  const double rev = load2(lam, b, t, o, im, ls, la);
  const i64 qx = t.jx << 2, qy = t.jy << 2;
  const i64 D = ls[1] + ls[3], A = ls[2] + ls[4];
  // the rows of the adjoint times rate/N: 8 A0 (kept at eight times for the
  // weights it enters with), 3 A1, 2 A2, 2 A3, 2 A4, 2 A5
  const i64 a8 = mulc(((D << 1) - A - (v0 << 2)) << 2, m.c[CM_E] << 1);
  const i64 b1 = mulc((v0 << 2) + D - (A << 1), m.c[CM_EPS]);
  const i64 n2 = mulc((la[1] - la[3]) + (la[4] << 1), m.c[CM_Q]);
  const i64 n3 = mulc((la[2] << 1) - (la[1] + la[3]), m.c[CM_Q]);
  const i64 h4 = mulc(ls[4] - ls[2], m.c[CM_P]);
  const i64 h5 = mulc(ls[3] - ls[1], m.c[CM_P]);
  // twice the gradient by j through the quadratic equilibria
  const i64 w = ((3 * a8 + 1) >> 1) - (b1 << 2);   // 2 (6 A0 - 2 (3 A1))
  const i64 gx = mulr(qx, (w + (h4 << 1)) << 1) + mulr(qy, h5 << 1);
  const i64 gy = mulr(qy, (w - (h4 << 1)) << 1) + mulr(qx, h5 << 1);
  i64 S[5], F[5];
  S[1] = ls[1] - a8 + h5;
  S[3] = ls[3] - a8 - h5;
  const i64 ax = (b1 << 1) - ((a8 + 2) >> 2);
  S[2] = ls[2] + ax + h4;
  S[4] = ls[4] + ax - h4;
  const i64 dx = gx - (n2 << 1), dy = gy - (n3 << 1);   // diagonals
  F[1] = la[1] + (dx - dy);
  F[3] = la[3] - (dx + dy);
  F[2] = la[2] - (gy + n3);
  F[4] = la[4] - (gx + n2);
  i64 f0 = (v0 << 1) + ((a8 + 1) >> 1) - (b1 << 1);
  src.add(S, F, f0);
  store2(S, F, f0, b, lam);
  return rev;
}

// ---------------------------------------------------------------------------
// D3Q19 BGK + partial bounce-back in pair form, completed by conservation as
// the D2Q9 one (pairs 1-3 the z, y, x axes, 4-5 the yz, 6-7 the xz, 8-9 the xy
// diagonals).  c[]: om/2, om/6.

struct Pairs3 {
  i64 s[10], a[10];
  i64 jx, jy, jz;
  __device__ __forceinline__ explicit Pairs3(const i64* x) {
    static_for<9>([&](auto D) {
      constexpr int d = decltype(D)::value + 1;
      s[d] = x[d] + x[d + 9];
      a[d] = x[d] - x[d + 9];
    });
    jx = ((a[9] - a[8]) + (a[7] - a[6])) - a[3];
    jy = ((a[5] - a[4]) - (a[8] + a[9])) - a[2];
    jz = -(((a[4] + a[5]) + (a[6] + a[7])) + a[1]);
  }
};

__device__ __forceinline__ void bgk3_odd(const Pairs3& t, const FixedModel& m, i64* o) {
  static_for<6>([&](auto D) {
    constexpr int d = decltype(D)::value + 4;
    o[d] = mulc(e_dot<LAT_D3Q19, d>(t.jx, t.jy, t.jz) - 6 * t.a[d], m.c[C2_SIXTH_OM]);
  });
  o[1] = -((o[4] + o[5]) + (o[6] + o[7]));
  o[2] = (o[5] - o[4]) - (o[8] + o[9]);
  o[3] = (o[7] - o[6]) + (o[9] - o[8]);
}

__device__ __forceinline__ void bgk3_collide(const i64* x, const Factor& im, const FixedModel& m,
                                             double* f) {
  const Pairs3 t(x);
  const i64* s = t.s;
  i64 o[10];
  bgk3_odd(t, m, o);
  const i64 qx = t.jx << 2, qy = t.jy << 2, qz = t.jz << 2;
  const i64 xx = sqr(qx), yy = sqr(qy), zz = sqr(qz);   // * 2^62
  const i64 xy = mulr(qx, qy) << 1, yz = mulr(qy, qz) << 1, xz = mulr(qx, qz) << 1;
  const i64 rho = x[0] + ((s[1] + s[2]) + s[3]) +
                  (((s[4] + s[5]) + (s[6] + s[7])) + (s[8] + s[9]));
  const i64 c = mulc(rho - ((3 * (xx + yy + zz)) >> 2), kEighteenth);
  // pair sums of the equilibrium: axes 2 c + (e.j)^2 / 2, diagonals c + (e.j)^2 / 4
  const i64 eq[10] = {0,
                      (c << 1) + (zz >> 2),
                      (c << 1) + (yy >> 2),
                      (c << 1) + (xx >> 2),
                      c + ((yy + zz + yz) >> 3),
                      c + ((yy + zz - yz) >> 3),
                      c + ((xx + zz + xz) >> 3),
                      c + ((xx + zz - xz) >> 3),
                      c + ((xx + yy + xy) >> 3),
                      c + ((xx + yy - xy) >> 3)};
  i64 left = 0;
  static_for<9>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    const i64 E = mulc((eq[d] - s[d]) << 1, m.c[C2_HALF_OM]);
    left += E;
    const i64 sp = s[d] + E;
    i64 ap = t.a[d] + o[d];
    ap -= im.times(ap << 1);
    f[d] = to_double(sp + ap, kScale + 1);
    f[d + 9] = to_double(sp - ap, kScale + 1);
  });
  f[0] = to_double((x[0] - left) << 1, kScale + 1);
}

// Transpose of bgk3_collide (see bgk2_reverse): 36 c0 = 12 lam_0 + 2 axes +
// diagonals, 12 c_a = q_a + j_a (3 P_aa - 36 c0) + 3 sum_b P_ab j_b, halved here.
__device__ __forceinline__ double bgk3_reverse(const i64* x, double* lam, const Block& b,
                                               const Factor& im, const FixedModel& m) {
  const Pairs3 t(x);
  i64 o[10], ls[10], la[10];
  bgk3_odd(t, m, o);
  PairDot rev;
  const i64 v0 = (b.load(lam[0]) + 8) >> 4;
  static_for<9>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    load_pair(b, lam[d], lam[d + 9], t.a[d] + o[d], im, ls[d], la[d], rev);
  });
  const i64 qx = t.jx << 2, qy = t.jy << 2, qz = t.jz << 2;
  const i64 dyz = ls[4] + ls[5], dxz = ls[6] + ls[7], dxy = ls[8] + ls[9];
  const i64 c36 = 12 * v0 + ((ls[1] + ls[2] + ls[3]) << 1) + (dyz + dxz + dxy);
  const i64 pxy = 3 * (ls[8] - ls[9]), pyz = 3 * (ls[4] - ls[5]), pxz = 3 * (ls[6] - ls[7]);
  const i64 ux = (la[9] - la[8]) + (la[7] - la[6]) - (la[3] << 1);
  const i64 uy = (la[5] - la[4]) - (la[8] + la[9]) - (la[2] << 1);
  const i64 uz = -((la[4] + la[5]) + (la[6] + la[7]) + (la[1] << 1));
  const i64 cx = ((ux + 1) >> 1) + mulr(qx, 3 * ((ls[3] << 1) + dxz + dxy) - c36) + mulr(qy, pxy) +
                 mulr(qz, pxz);
  const i64 cy = ((uy + 1) >> 1) + mulr(qy, 3 * ((ls[2] << 1) + dyz + dxy) - c36) + mulr(qx, pxy) +
                 mulr(qz, pyz);
  const i64 cz = ((uz + 1) >> 1) + mulr(qz, 3 * ((ls[1] << 1) + dyz + dxz) - c36) + mulr(qx, pxz) +
                 mulr(qy, pyz);
  const u64 h3 = m.c[C2_SIXTH_OM] << 1, h18 = m.c[C2_SIXTH_OM] / 3;
  lam[0] = b.store((v0 << 1) + mulc(c36 - 36 * v0, h18));
  static_for<9>([&](auto D) {
    constexpr int d = decltype(D)::value + 1;
    const i64 S = ls[d] + mulc(c36 - 18 * ls[d], h18);
    const i64 F = la[d] + mulc(e_dot<LAT_D3Q19, d>(cx, cy, cz) - 3 * la[d], h3);
    lam[d] = b.store(S + F);
    lam[d + 9] = b.store(S - F);
  });
  return rev.value(b);
}

// ---------------------------------------------------------------------------
// Temperature lattice (D2Q5: 1, 3 the y and 2, 4 the x pair).  Temperatures have
// no known size, so the cell's five populations carry a scale of their own; the
// populations are linear in it.  om6: om_T / 6 * 2^64.  The solid's heating
// source is added in FP64, where there is any.

using ThermalBlock = BlockOf<58>;

// T and 3 T u of the populations g (in a Block's units)
struct Thermal {
  i64 g[5], T, tx, ty;
  __device__ __forceinline__ Thermal(const double* gp, const ThermalBlock& b, i64 jx, i64 jy) {
    static_for<5>([&](auto I) { g[decltype(I)::value] = b.load(gp[decltype(I)::value]); });
    T = g[0] + ((g[1] + g[3]) + (g[2] + g[4]));
    tx = 3 * mulr(jx << 2, T << 1);
    ty = 3 * mulr(jy << 2, T << 1);
  }
  // 6 (g_eq - g) of direction i, the rest direction's 3 (g_eq - g)
  template <int i>
  __device__ __forceinline__ i64 excess() const {
    if constexpr (i == 0) return T - 3 * g[0];
    if constexpr (i == 1) return T - ty - 6 * g[1];
    if constexpr (i == 2) return T - tx - 6 * g[2];
    if constexpr (i == 3) return T + ty - 6 * g[3];
    if constexpr (i == 4) return T + tx - 6 * g[4];
  }
};

__device__ __forceinline__ void thermal_collide(const Thermal& t, const ThermalBlock& b, u64 om6,
                                                double* gp) {
  i64 left = 0;
  static_for<4>([&](auto I) {
    constexpr int i = decltype(I)::value + 1;
    const i64 d = mulc(t.template excess<i>(), om6);
    left += d;
    gp[i] = to_double(t.g[i] + d, b.k);
  });
  gp[0] = to_double(t.g[0] - left, b.k);
}

// Transpose: lam[0..4] in and out (without the heating term); l the adjoint's
// own scale.  dx, dy: lam_4 - lam_2 and lam_3 - lam_1, sum6: 2 lam_0 + the others
// (both before the collision).
struct ThermalAdjoint {
  double dx, dy, sum6;
};
__device__ __forceinline__ ThermalAdjoint thermal_reverse(double* lam, const ThermalBlock& l, i64 jx,
                                                          i64 jy, u64 om6) {
  i64 v[5];
  static_for<5>([&](auto I) { v[decltype(I)::value] = l.load(lam[decltype(I)::value]); });
  const i64 dx = v[4] - v[2], dy = v[3] - v[1];
  const i64 s6 = (v[0] << 1) + ((v[1] + v[3]) + (v[2] + v[4]));
  const i64 c6 = s6 + 3 * (mulr(jx << 2, dx << 1) + mulr(jy << 2, dy << 1));
  static_for<5>([&](auto I) {
    constexpr int i = decltype(I)::value;
    lam[i] = to_double(v[i] + mulc(c6 - 6 * v[i], om6), l.k);
  });
  return ThermalAdjoint{to_double(dx, l.k), to_double(dy, l.k), to_double(s6, l.k)};
}

// ---------------------------------------------------------------------------
// The dissipation objective on the 2D lattices (ObjDissipation): second
// moments free of the equilibrium, V_ab = sum e_a e_b f - rho/3 - j_a j_b.

struct Stress2 {
  i64 xx, yy, xy;   // * 2^61
  i64 qx, qy;       // j * 2^63
  __device__ __forceinline__ Stress2(const i64* x, const Pairs2& t) {
    constexpr u64 kThird = 0x5555555555555556ull;
    qx = t.jx << 2;
    qy = t.jy << 2;
    const i64 a = sqr(qx), b = sqr(qy);
    const i64 D = t.s[1] + t.s[3];
    const i64 third = mulc((x[0] + D) + (t.s[2] + t.s[4]), kThird);
    xx = D + t.s[4] - third - (a >> 1);
    yy = D + t.s[2] - third - (b >> 1);
    xy = t.s[3] - t.s[1] - (mulr(qx, qy) >> 1);
  }
  // j^2 in FP64: a slow flow's square needs its own exponent
  __device__ __forceinline__ double jj() const {
    const double x = to_double(qx, 63), y = to_double(qy, 63);
    return x * x + y * y;
  }
};

__device__ __forceinline__ u128 square(i64 a) {
  const u64 m = (u64)(a.negative() ? -a : a);
  return (u128)m * m;
}
// a * c / 2^64
__device__ __forceinline__ u128 times(u128 a, u64 c) {
  return (u128)(u64)(a >> 64) * c + (u64)(((u128)(u64)a * c) >> 64);
}

// (2 alpha j^2 + cv V:V) * 2^117, cv given * 2^64: below 2^121.  The 128-bit
// products leave a slow flow's squares (1e-14 at u = 1e-7) their bits, and cost
// four 32-bit multiplies of 1.4 cycles a warp each where a conversion or a
// product on the FP64 pipe takes 16.
constexpr int kEnergyScale = 117;
__device__ __forceinline__ u128 dissipation2(const i64* x, u64 im, u64 cv) {
  const Stress2 v(x, Pairs2(x));
  const u128 a = times(square(v.qx) + square(v.qy), im);               // * 2^126
  const u128 b = times(square(v.xx) + square(v.yy) + 2 * square(v.xy), cv);   // * 2^122
  return (a >> (126 - 1 - kEnergyScale)) + (b >> (122 - kEnergyScale));
}
__device__ __forceinline__ double energy(u128 e) {
  u64 h = (u64)(e >> 64), l = (u64)e;
  int k = kEnergyScale - 64;
  if (h == 0ull) {
    h = l;
    l = 0ull;
    k += 64;
  }
  if (h == 0ull) return 0.;
  const int s = clz64(h) - 1;   // as a positive i64
  h = s >= 0 ? (h << s) | ((l >> 1) >> (63 - s)) : h >> 1;
  return to_double((i64)h, k + s);
}

// The objective's derivatives by f and by imult, both over the weight.
struct Dissipation2 {
  Source2 src;    // * 2^61
  double dim;     // 2 j^2
  // c: cv * 2^64
  __device__ __forceinline__ Dissipation2(const i64* x, const Factor& im, u64 c) {
    const Stress2 v(x, Pairs2(x));
    constexpr u64 kThird = 0x5555555555555556ull;
    const i64 t3 = mulc(v.xx + v.yy, kThird);
    // V j
    const i64 vx = mulr(v.qx, v.xx << 1) + mulr(v.qy, v.xy << 1);
    const i64 vy = mulr(v.qx, v.xy << 1) + mulr(v.qy, v.yy << 1);
    // 4 (alpha j - cv V j) along e, 2 cv (e.V e - tr/3) even
    src.gx = im.times(v.qx) - (mulc(vx, c) << 2);
    src.gy = im.times(v.qy) - (mulc(vy, c) << 2);
    const i64 d = v.xx + v.yy - t3, s = v.xy << 1;
    src.ev[0] = -mulc(t3 << 1, c);
    src.ev[1] = mulc((d - s) << 1, c);
    src.ev[2] = mulc((v.yy - t3) << 1, c);
    src.ev[3] = mulc((d + s) << 1, c);
    src.ev[4] = mulc((v.xx - t3) << 1, c);
    dim = 2. * v.jj();
  }
  // The finest scale of a Block whose units take the source times the weight
  // (scaled): its error, some units of w 2^-61, is far above 2^-89 w.  Where the
  // adjoint is much smaller than the source (the first reverse steps, a fluid at
  // rest) its own finer units would not: with an FP64 sum for such cells a
  // 2048x1024 reverse step whose flow has not developed takes 200 us against 141.
  __device__ __forceinline__ int scale_limit(const FixedModel& m) const {
    const i64 v[7] = {src.ev[0], src.ev[1], src.ev[2], src.ev[3], src.ev[4], src.gx, src.gy};
    u64 any = 1u;
    static_for<7>([&](auto I) {
      const i64 t = v[decltype(I)::value];
      any |= (u64)(t ^ (t >> 63));
    });
    const int sh = clz64(any) - 5;   // one bit for the product's rounding
    return 64 - m.w_exp + (sh < 27 ? sh : 27);
  }
  // the source times the weight in the units of a Block's results, where that
  // fits (on)
  __device__ __forceinline__ Source2 scaled(const FixedModel& m, const Block& b) const {
    Source2 r;
    const int sh = m.w_exp + b.k - 64;
    i64 v[7] = {src.ev[0], src.ev[1], src.ev[2], src.ev[3], src.ev[4], src.gx, src.gy};
    u64 any = 0u;
    static_for<7>([&](auto I) {
      i64& t = v[decltype(I)::value];
      t = mulc(t, m.w);
      any |= (u64)(t ^ (t >> 63));
    });
    r.on = !b.zero && b.ok && sh < 28 && (sh <= 0 || (any >> (60 - sh)) == 0u);
    const int l = sh > 0 ? sh : 0, q = sh < 0 ? (sh > -63 ? -sh : 63) : 0;
    const i64 half = q > 0 ? 1ll << (q - 1) : 0, neg = m.w_neg;
    static_for<7>([&](auto I) {
      i64& t = v[decltype(I)::value];
      t = ((t << l) + half) >> q;
      t = (t ^ neg) - neg;
    });
    static_for<5>([&](auto I) { r.ev[decltype(I)::value] = v[decltype(I)::value]; });
    r.gx = v[5];
    r.gy = v[6];
    return r;
  }
};

// f <- the flow collision of LAT and COLL.
template <int LAT, int COLL>
__device__ __forceinline__ void collide(const i64* x, const Factor& im, const FixedModel& m,
                                        double* f) {
  if constexpr (LAT == LAT_D3Q19 && COLL == LBM_MRT) mrt3d_collide(x, im, m, f);
  if constexpr (LAT == LAT_D3Q19 && COLL == LBM_BGK) bgk3_collide(x, im, m, f);
  if constexpr (LAT != LAT_D3Q19 && COLL == LBM_BGK) bgk2_collide(x, im, m, f);
  if constexpr (LAT == LAT_D2Q9 && COLL == LBM_MRT) mrt2_collide(x, im, m, f);
}

// lam <- its transpose (plus src on the 2D lattices); returns the derivative by
// imult.
template <int LAT, int COLL>
__device__ __forceinline__ double reverse(const i64* x, double* lam, const Block& b,
                                          const Factor& im, const FixedModel& m,
                                          const Source2& src) {
  if constexpr (LAT == LAT_D3Q19 && COLL == LBM_MRT) return mrt3d_reverse(x, lam, b, im, m);
  if constexpr (LAT == LAT_D3Q19 && COLL == LBM_BGK) return bgk3_reverse(x, lam, b, im, m);
  if constexpr (LAT != LAT_D3Q19 && COLL == LBM_BGK) return bgk2_reverse(x, lam, b, im, m, src);
  if constexpr (LAT == LAT_D2Q9 && COLL == LBM_MRT) return mrt2_reverse(x, lam, b, im, m, src);
}

}  // namespace fx
}  // namespace lbm
