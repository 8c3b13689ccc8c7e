// Exact-arithmetic helpers shared by the sm_100a kernels and the host-side
// self-tests: IEEE-754 binary64 operations with no contraction, double-double
// arithmetic, a near-correctly-rounded sin/cos for the ray-direction angle, and
// the 128-bit PCG64 (XSL-RR 128/64) generator that NumPy's PCG64 implements.
//
// Every function here compiles both as CUDA device code and as plain C++ on the
// host (g++ -ffp-contract=off), so the host tests exercise the very same code the
// kernels run.
#pragma once
#include <stdint.h>
#include <math.h>

#if defined(__CUDACC__)
#define PR_HD __host__ __device__ __forceinline__
#else
#define PR_HD static inline
#endif

// ---------------------------------------------------------------------------
// Binary64 primitives. On the device these are the round-to-nearest intrinsics,
// which the compiler never fuses into FMAs; on the host the file is compiled with
// -ffp-contract=off so the plain operators mean the same thing.
// ---------------------------------------------------------------------------
PR_HD double pr_add(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
PR_HD double pr_sub(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dsub_rn(a, b);
#else
  return a - b;
#endif
}
PR_HD double pr_mul(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
PR_HD double pr_div(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __ddiv_rn(a, b);
#else
  return a / b;
#endif
}
PR_HD double pr_sqrt(double a) {
#if defined(__CUDA_ARCH__)
  return __dsqrt_rn(a);
#else
  return sqrt(a);
#endif
}
PR_HD double pr_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return fma(a, b, c);
#endif
}

// NumPy's float64 remainder for a positive divisor: the sign of the result follows
// the divisor (Python semantics); fmod is exact, the correction is one rounded add.
PR_HD double pr_pymod_pos(double a, double b) {
  double m = fmod(a, b);
  if (m != 0.0) {
    if (m < 0.0) m = pr_add(m, b);
  } else {
    m = 0.0;  // +0.0, the sign of the divisor
  }
  return m;
}

// ---------------------------------------------------------------------------
// Double-double arithmetic (Dekker / Knuth error-free transforms, FMA products).
// ---------------------------------------------------------------------------
struct pr_dd {
  double hi, lo;
};

PR_HD pr_dd pr_two_sum(double a, double b) {
  double s = pr_add(a, b);
  double bb = pr_sub(s, a);
  double e = pr_add(pr_sub(a, pr_sub(s, bb)), pr_sub(b, bb));
  return {s, e};
}
PR_HD pr_dd pr_fast_two_sum(double a, double b) {  // requires |a| >= |b| or a == 0
  double s = pr_add(a, b);
  double e = pr_sub(b, pr_sub(s, a));
  return {s, e};
}
PR_HD pr_dd pr_two_prod(double a, double b) {
  double p = pr_mul(a, b);
  double e = pr_fma(a, b, -p);
  return {p, e};
}
PR_HD pr_dd pr_dd_mul(pr_dd a, pr_dd b) {
  pr_dd p = pr_two_prod(a.hi, b.hi);
  double e = pr_add(p.lo, pr_add(pr_mul(a.hi, b.lo), pr_mul(a.lo, b.hi)));
  return pr_fast_two_sum(p.hi, e);
}
PR_HD pr_dd pr_dd_mul_d(pr_dd a, double b) {
  pr_dd p = pr_two_prod(a.hi, b);
  double e = pr_fma(a.lo, b, p.lo);
  return pr_fast_two_sum(p.hi, e);
}
PR_HD pr_dd pr_dd_add(pr_dd a, pr_dd b) {
  pr_dd s = pr_two_sum(a.hi, b.hi);
  pr_dd t = pr_two_sum(a.lo, b.lo);
  double e = pr_add(s.lo, t.hi);
  s = pr_fast_two_sum(s.hi, e);
  e = pr_add(s.lo, t.lo);
  return pr_fast_two_sum(s.hi, e);
}

// ---------------------------------------------------------------------------
// sin and cos of x in [0, 2*pi] (the Lambertian azimuth 2*pi*u).
//
// Method: Cody-Waite reduction r = x - k*pi/2 with pi/2 split into a 33-bit, a
// 33-bit and a 53-bit part (k <= 4, so k*P1 and k*P2 are exact and x - k*P1 is
// exact by Sterbenz' lemma), carried as a double-double; then the Taylor series
// of sin and cos about 0 for |r| <= pi/4, with the low-order coefficients in
// double-double and the tail (relative size < 1e-6) in binary64 Horner form.
// The double-double result carries a relative error below about 2^-70, so its
// rounding to binary64 is the correctly rounded value except when the exact value
// lies within that distance of a rounding midpoint.
//
// The constants are the binary64 (or double-double) roundings of pi/2 pieces and
// of (-1)^n / n!, computed exactly with rational arithmetic.
// ---------------------------------------------------------------------------
#define PR_PIO2_1 0x1.921fb54400000p+0    // pi/2 truncated to 33 bits
#define PR_PIO2_2 0x1.0b4611a600000p-34   // next 33 bits
#define PR_PIO2_3 0x1.3198a2e037073p-69   // remainder rounded to 53 bits
#define PR_TWO_OVER_PI 0x1.45f306dc9c883p-1

PR_HD void pr_sincos_reduced(pr_dd r, double* s_out, double* c_out) {
  const pr_dd z = pr_dd_mul(r, r);
  const double zh = z.hi;
  // sin(r) = r + r*z*(s3 + z*(s5 + z*(s7 + z*T(z)))),  T(z) = s9 + s11 z + ... + s21 z^6
  double ts = 0x1.71b8ef6dcf572p-66;              // 1/21!
  ts = pr_fma(ts, zh, -0x1.2f49b46814157p-57);   // -1/19!
  ts = pr_fma(ts, zh, 0x1.952c77030ad4ap-49);    // 1/17!
  ts = pr_fma(ts, zh, -0x1.ae7f3e733b81fp-41);   // -1/15!
  ts = pr_fma(ts, zh, 0x1.6124613a86d09p-33);    // 1/13!
  ts = pr_fma(ts, zh, -0x1.ae64567f544e4p-26);   // -1/11!
  ts = pr_fma(ts, zh, 0x1.71de3a556c734p-19);    // 1/9!
  pr_dd qs = pr_dd_add(pr_dd{-0x1.a01a01a01a01ap-13, -0x1.a01a01a01a01ap-73}, pr_dd_mul_d(z, ts));  // s7
  qs = pr_dd_add(pr_dd{0x1.1111111111111p-7, 0x1.1111111111111p-63}, pr_dd_mul(z, qs));           // s5
  qs = pr_dd_add(pr_dd{-0x1.5555555555555p-3, -0x1.5555555555555p-57}, pr_dd_mul(z, qs));         // s3
  pr_dd sn = pr_dd_add(r, pr_dd_mul(pr_dd_mul(r, z), qs));
  // cos(r) = 1 + z*(-1/2 + z*(c4 + z*(c6 + z*(c8 + z*U(z))))),  U(z) = c10 + ... + c22 z^6
  double tc = -0x1.0ce396db7f853p-70;             // -1/22!
  tc = pr_fma(tc, zh, 0x1.e542ba4020225p-62);    // 1/20!
  tc = pr_fma(tc, zh, -0x1.6827863b97d97p-53);   // -1/18!
  tc = pr_fma(tc, zh, 0x1.ae7f3e733b81fp-45);    // 1/16!
  tc = pr_fma(tc, zh, -0x1.93974a8c07c9dp-37);   // -1/14!
  tc = pr_fma(tc, zh, 0x1.1eed8eff8d898p-29);    // 1/12!
  tc = pr_fma(tc, zh, -0x1.27e4fb7789f5cp-22);   // -1/10!
  pr_dd qc = pr_dd_add(pr_dd{0x1.a01a01a01a01ap-16, 0x1.a01a01a01a01ap-76}, pr_dd_mul_d(z, tc));  // c8
  qc = pr_dd_add(pr_dd{-0x1.6c16c16c16c17p-10, 0x1.f49f49f49f49fp-65}, pr_dd_mul(z, qc));         // c6
  qc = pr_dd_add(pr_dd{0x1.5555555555555p-5, 0x1.5555555555555p-59}, pr_dd_mul(z, qc));           // c4
  qc = pr_dd_add(pr_dd{-0.5, 0.0}, pr_dd_mul(z, qc));
  pr_dd cs = pr_dd_add(pr_dd{1.0, 0.0}, pr_dd_mul(z, qc));
  *s_out = sn.hi;
  *c_out = cs.hi;
}

PR_HD void pr_sincos(double x, double* s_out, double* c_out) {
  const double kd = rint(pr_mul(x, PR_TWO_OVER_PI));
  const int k = (int)kd;
  // r = x - k*(P1 + P2 + P3) as a double-double
  const double r1 = pr_sub(x, pr_mul(kd, PR_PIO2_1));  // exact
  pr_dd r = pr_two_sum(r1, -pr_mul(kd, PR_PIO2_2));     // k*P2 exact
  r = pr_fast_two_sum(r.hi, pr_sub(r.lo, pr_mul(kd, PR_PIO2_3)));
  double s, c;
  pr_sincos_reduced(r, &s, &c);
  switch (k & 3) {
    case 0: *s_out = s; *c_out = c; break;
    case 1: *s_out = c; *c_out = -s; break;
    case 2: *s_out = -s; *c_out = -c; break;
    default: *s_out = -c; *c_out = s; break;
  }
}

// ---------------------------------------------------------------------------
// The same sin and cos, bit for bit, for x in [0, 2 pi], from a table and a rounding test
// (table-driven evaluation as in Gal, "Computing elementary functions", 1986, and Ziv's test,
// "Fast evaluation of elementary mathematical functions with correctly rounded last bit",
// 1991).  x = k pi/64 + r with |r| <= pi/128; S_k = sin(k pi/64) and C_k = S_{k+32} are
// double-double table values, and
//   sin x = S + C r - S z/2 + [C (sin r - r) + S (cos r - 1 + z/2)],  z = r r,
//   cos x = C - S r - C z/2 - [S (sin r - r) - C (cos r - 1 + z/2)],
// the first three terms in double-double, the bracket (below 2.6e-6) in binary64.  Every
// operation on the bracket's terms c and d rounds by 2^-53 of them, fewer than 16 in all, so the
// result h + l is within E = 2^-48.8 (|c| + |d|) + 2^-68 |h| of the exact value; the last term
// also covers the error of the double-double series above.  When h + (l - E) and h + (l + E)
// round alike, both evaluations round to that value; else the series decides (about one ray in
// 10^4).  The series costs about 330 binary64 operations a ray, this 100.
// ---------------------------------------------------------------------------
struct pr_sin_table {
  double v[322];  // (hi, lo) of sin(k pi/64), k = 0 .. 160
};
constexpr double kPrSinQuadrant[33][2] = {
    {0.0, 0.0},
    {0x1.91f65f10dd814p-5, -0x1.912bd0d569a90p-61},
    {0x1.917a6bc29b42cp-4, -0x1.e2718d26ed688p-60},
    {0x1.2c8106e8e613ap-3, 0x1.13000a89a11e0p-58},
    {0x1.8f8b83c69a60bp-3, -0x1.26d19b9ff8d82p-57},
    {0x1.f19f97b215f1bp-3, -0x1.42deef11da2c4p-57},
    {0x1.294062ed59f06p-2, -0x1.5d28da2c4612dp-56},
    {0x1.58f9a75ab1fddp-2, -0x1.efdc0d58cf620p-62},
    {0x1.87de2a6aea963p-2, -0x1.72cedd3d5a610p-57},
    {0x1.b5d1009e15cc0p-2, 0x1.5b362cb974183p-57},
    {0x1.e2b5d3806f63bp-2, 0x1.e0d891d3c6841p-58},
    {0x1.073879922ffeep-1, -0x1.a5a014347406cp-55},
    {0x1.1c73b39ae68c8p-1, 0x1.b25dd267f6600p-55},
    {0x1.30ff7fce17035p-1, -0x1.efcc626f74a6fp-57},
    {0x1.44cf325091dd6p-1, 0x1.8076a2cfdc6b3p-57},
    {0x1.57d69348ceca0p-1, -0x1.75720992bfbb2p-55},
    {0x1.6a09e667f3bcdp-1, -0x1.bdd3413b26456p-55},
    {0x1.7b5df226aafafp-1, -0x1.0f537acdf0ad7p-56},
    {0x1.8bc806b151741p-1, -0x1.2c5e12ed1336dp-55},
    {0x1.9b3e047f38741p-1, -0x1.30ee286712474p-55},
    {0x1.a9b66290ea1a3p-1, 0x1.9f630e8b6dac8p-60},
    {0x1.b728345196e3ep-1, -0x1.bc69f324e6d61p-55},
    {0x1.c38b2f180bdb1p-1, -0x1.6e0b1757c8d07p-56},
    {0x1.ced7af43cc773p-1, -0x1.e7b6bb5ab58aep-58},
    {0x1.d906bcf328d46p-1, 0x1.457e610231ac2p-56},
    {0x1.e212104f686e5p-1, -0x1.014c76c126527p-55},
    {0x1.e9f4156c62ddap-1, 0x1.760b1e2e3f81ep-55},
    {0x1.f0a7efb9230d7p-1, 0x1.52c7adc6b4989p-56},
    {0x1.f6297cff75cb0p-1, 0x1.562172a361fd3p-56},
    {0x1.fa7557f08a517p-1, -0x1.7a0a8ca13571fp-55},
    {0x1.fd88da3d12526p-1, -0x1.87df6378811c7p-55},
    {0x1.ff621e3796d7ep-1, -0x1.c57bc2e24aa15p-57},
    {0x1.0000000000000p+0, 0x0.0p+0},
};
constexpr pr_sin_table pr_make_sin_table() {
  pr_sin_table t{};
  for (int k = 0; k <= 160; ++k) {
    const int m = k & 63;                     // sin(pi + a) = -sin a
    const int q = m <= 32 ? m : 64 - m;       // sin(pi - a) = sin a
    const double sign = (k & 64) ? -1.0 : 1.0;
    t.v[2 * k] = sign * kPrSinQuadrant[q][0];
    t.v[2 * k + 1] = sign * kPrSinQuadrant[q][1];
  }
  return t;
}
#if defined(__CUDACC__)
static __device__ const pr_sin_table g_pr_sin_table = pr_make_sin_table();
#endif
#if !defined(__CUDA_ARCH__)
static constexpr pr_sin_table k_pr_sin_table_host = pr_make_sin_table();
#endif

#define PR_PI64_1 0x1.921fb54400000p-5    // pi/64 truncated to 33 bits
#define PR_PI64_2 0x1.0b4611a600000p-39   // next 33 bits
#define PR_PI64_3 0x1.3198a2e037073p-74   // remainder rounded to 53 bits
#define PR_64_OVER_PI 0x1.45f306dc9c883p+4

// One of the two sums above: T + A r + B z/2 (A, B, T double-double; w = B / 2), bracket c + d.
// Returns false when the rounding is not decided.
PR_HD bool pr_ziv_sum(double th, double tl, double ah, double al, double wh, double wl, double rh, double rl,
                      double zh, double zl, double c, double d, double* out) {
  const double a = pr_mul(ah, rh);
  const double ae = pr_fma(al, rh, pr_fma(ah, rl, pr_fma(ah, rh, -a)));
  const double b = pr_mul(wh, zh);
  const double be = pr_fma(wl, zh, pr_fma(wh, zl, pr_fma(wh, zh, -b)));
  const pr_dd s1 = pr_two_sum(th, a);
  const pr_dd s2 = pr_fast_two_sum(s1.hi, b);
  const double low = pr_add(pr_add(pr_add(s1.lo, s2.lo), tl), pr_add(ae, be));
  const double l = pr_add(low, pr_add(c, d));
  const double e = pr_fma(pr_add(fabs(c), fabs(d)), 0x1.3p-49, pr_mul(fabs(s2.hi), 0x1.0p-68));
  const double up = pr_add(s2.hi, pr_add(l, e)), dn = pr_add(s2.hi, pr_sub(l, e));
  *out = up;
  return up == dn;
}

PR_HD void pr_sincos_2pi(double x, double* s_out, double* c_out) {
  const double kd = rint(pr_mul(x, PR_64_OVER_PI));
  const int k = (int)kd;  // 0 .. 128
  const double r1 = pr_sub(x, pr_mul(kd, PR_PI64_1));  // both exact
  pr_dd r = pr_two_sum(r1, -pr_mul(kd, PR_PI64_2));     // k P2 exact
  r = pr_fast_two_sum(r.hi, pr_sub(r.lo, pr_mul(kd, PR_PI64_3)));
#if defined(__CUDA_ARCH__)
  const double2 S = __ldg(reinterpret_cast<const double2*>(g_pr_sin_table.v) + k);
  const double2 C = __ldg(reinterpret_cast<const double2*>(g_pr_sin_table.v) + k + 32);
  const double sh = S.x, sl = S.y, ch = C.x, cl = C.y;
#else
  const double* T = k_pr_sin_table_host.v;
  const double sh = T[2 * k], sl = T[2 * k + 1], ch = T[2 * k + 64], cl = T[2 * k + 65];
#endif
  const double zh = pr_mul(r.hi, r.hi);
  const double zl = pr_fma(pr_add(r.hi, r.hi), r.lo, pr_fma(r.hi, r.hi, -zh));
  // sin r - r and cos r - 1 + z/2 (Taylor; the next terms are below 2^-72 of r and 2^-80)
  double p = pr_fma(zh, 0x1.71de3a556c734p-19, -0x1.a01a01a01a01ap-13);
  p = pr_fma(zh, p, 0x1.1111111111111p-7);
  p = pr_fma(zh, p, -0x1.5555555555555p-3);
  const double sm = pr_mul(pr_mul(r.hi, zh), p);
  double q = pr_fma(zh, -0x1.27e4fb7789f5cp-22, 0x1.a01a01a01a01ap-16);
  q = pr_fma(zh, q, -0x1.6c16c16c16c17p-10);
  q = pr_fma(zh, q, 0x1.5555555555555p-5);
  const double cm = pr_mul(pr_mul(zh, zh), q);
  const bool s_ok = pr_ziv_sum(sh, sl, ch, cl, -0.5 * sh, -0.5 * sl, r.hi, r.lo, zh, zl, pr_mul(ch, sm),
                               pr_mul(sh, cm), s_out);
  const bool c_ok = pr_ziv_sum(ch, cl, -sh, -sl, -0.5 * ch, -0.5 * cl, r.hi, r.lo, zh, zl, -pr_mul(sh, sm),
                               pr_mul(ch, cm), c_out);
  if (!(s_ok && c_ok)) pr_sincos(x, s_out, c_out);
}

// ---------------------------------------------------------------------------
// Correctly rounded quotients from a correctly rounded reciprocal (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990): with y = RN(1/b) and q one
// of the two binary64 neighbours of a/b, the remainder a - b q is exact and RN(q + y (a - b q)) is
// RN(a/b).  RN(a y) may be two units off, so one such step makes q a neighbour and the second
// rounds it.  For operands far from overflow and underflow (the traversal's: b in [2^-90, 1], a in
// [2^-60, 2] or 0).
// ---------------------------------------------------------------------------
PR_HD double pr_rcp(double b) {
#if defined(__CUDA_ARCH__)
  return __drcp_rn(b);
#else
  return 1.0 / b;
#endif
}
PR_HD double pr_div_rcp(double a, double b, double y) {
  double q = pr_mul(a, y);
  q = pr_fma(pr_fma(-b, q, a), y, q);
  return pr_fma(pr_fma(-b, q, a), y, q);
}

PR_HD int64_t pr_double_bits(double v) {
#if defined(__CUDA_ARCH__)
  return (int64_t)__double_as_longlong(v);
#else
  union { double d; int64_t i; } u;
  u.d = v;
  return u.i;
#endif
}
PR_HD double pr_bits_double(int64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  union { double d; int64_t i; } u;
  u.i = b;
  return u.d;
#endif
}

// (x, y, z) divided by sqrt((x x + y y) + z z), every operation rounded to nearest, for a vector
// of unit length up to its components' roundings.  The sum of squares is then s = 1 + k 2^-52
// (k >= 0) or 1 + k 2^-53 (k < 0) with a small integer k, the difference of the bit patterns of s
// and 1, and sqrt(s) = 1 + k/2 units - k^2/8 units^2 ...: never a tie, rounded to 1 + floor(k/2)
// units on either side.  With len = 1 + L units, RN(1/len) is 1 - 2 L units of 2^-53 (L >= 0) or
// 1 + ceil(-L/2) units of 2^-52 (L < 0), and v - (len - 1) v rounds to a neighbour of v/len, so
// one Markstein step gives RN(v/len).  Other lengths take the square root and the divisions.
PR_HD void pr_unit_vector(double* x, double* y, double* z) {
  const double s = pr_add(pr_add(pr_mul(*x, *x), pr_mul(*y, *y)), pr_mul(*z, *z));
  const int64_t one = 0x3ff0000000000000ll;
  const int64_t k = pr_double_bits(s) - one;
  if (k >= -1024 && k <= 1024) {
    const int64_t L = k >> 1;
    const double len = pr_bits_double(one + L);
    const double inv = pr_bits_double(L >= 0 ? one - 2 * L : one + ((1 - L) >> 1));
    const double d = pr_sub(len, 1.0);  // exact
    double q = pr_fma(-d, *x, *x);
    *x = pr_fma(pr_fma(-q, len, *x), inv, q);
    q = pr_fma(-d, *y, *y);
    *y = pr_fma(pr_fma(-q, len, *y), inv, q);
    q = pr_fma(-d, *z, *z);
    *z = pr_fma(pr_fma(-q, len, *z), inv, q);
    return;
  }
  const double len = pr_sqrt(s);
  *x = pr_div(*x, len);
  *y = pr_div(*y, len);
  *z = pr_div(*z, len);
}

// ---------------------------------------------------------------------------
// PCG64 (PCG XSL-RR 128/64, the generator behind numpy.random.PCG64):
//   state <- state * M + inc (mod 2^128), then output = rotr64(hi ^ lo, hi >> 58).
// A jump of n steps is the affine map state <- A_n state + C_n; the host supplies
// the maps for n = 2^0 .. 2^63 of a given stream.
// ---------------------------------------------------------------------------
struct pr_u128 {
  uint64_t lo, hi;
};

PR_HD uint64_t pr_umulhi64(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * (unsigned __int128)b) >> 64);
#endif
}
PR_HD pr_u128 pr_u128_mul(pr_u128 a, pr_u128 b) {  // low 128 bits of a*b
  pr_u128 r;
  r.lo = a.lo * b.lo;
  r.hi = pr_umulhi64(a.lo, b.lo) + a.hi * b.lo + a.lo * b.hi;
  return r;
}
PR_HD pr_u128 pr_u128_add(pr_u128 a, pr_u128 b) {
  pr_u128 r;
  r.lo = a.lo + b.lo;
  r.hi = a.hi + b.hi + (r.lo < a.lo ? 1u : 0u);
  return r;
}
PR_HD pr_u128 pr_u128_affine(pr_u128 mul, pr_u128 add, pr_u128 s) {
  return pr_u128_add(pr_u128_mul(mul, s), add);
}

#define PR_PCG_MULT_HI 0x2360ED051FC65DA4ull
#define PR_PCG_MULT_LO 0x4385DF649FCCF645ull

PR_HD uint64_t pr_pcg_output(pr_u128 s) {
  const uint64_t v = s.hi ^ s.lo;
  const unsigned rot = (unsigned)(s.hi >> 58);
#if defined(__CUDA_ARCH__)
  // rotate right by rot: the halves change places from 32 on, then two funnel shifts by rot mod 32
  const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
  const uint32_t a = rot & 32u ? hi : lo, b = rot & 32u ? lo : hi;
  return ((uint64_t)__funnelshift_r(b, a, rot) << 32) | __funnelshift_r(a, b, rot);
#else
  return (v >> rot) | (v << ((64u - rot) & 63u));
#endif
}

// One PCG64 draw mapped to [0, 1) the way numpy.random.Generator.random does:
// the top 53 bits times 2^-53.
PR_HD double pr_pcg_next_double(pr_u128* s, pr_u128 inc) {
  const pr_u128 m = {PR_PCG_MULT_LO, PR_PCG_MULT_HI};
  *s = pr_u128_affine(m, inc, *s);
  const uint64_t v = pr_pcg_output(*s) >> 11;
#if defined(__CUDA_ARCH__)
  // the same value by two exact sums: 2^31 + (v >> 32) 2^-21 and 0.5 + (v mod 2^32) 2^-53
  const double hi = __hiloint2double(0x41e00000, (int)(v >> 32)), lo = __hiloint2double(0x3fe00000, (int)(uint32_t)v);
  return pr_add(pr_sub(hi, 0x1.0p31 + 0.5), lo);
#else
  return (double)v * 0x1.0p-53;
#endif
}

// Jump a stream ahead by n steps using the power-of-two maps table[2*i] = A_{2^i},
// table[2*i + 1] = C_{2^i}.
PR_HD pr_u128 pr_pcg_jump(pr_u128 s, uint64_t n, const pr_u128* table) {
  int i = 0;
  while (n) {
    if (n & 1u) s = pr_u128_affine(table[2 * i], table[2 * i + 1], s);
    n >>= 1;
    ++i;
  }
  return s;
}
