// stx_rates.cuh -- the logarithm and the Arrhenius form of the packed reaction
// records, in two doubles.  Plain C++ besides the qualifiers, so that they are
// tested on the host against exact values; compile without FMA contraction.
#pragma once
#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define STX_HD __host__ __device__ __forceinline__
#else
#define STX_HD inline
#endif

// ln 2 in two parts, the first with 32 significant bits (e LN2_HI is exact for any exponent e)
#define LN2_HI 0x1.62e42feep-1
#define LN2_LO 0x1.a39ef35793c76p-33

// ln x as hi + lo, for 1 <= x <= 1e6 (any normal x > 0 works): x = 2^e m,
// ln m = 2 atanh(s), s = (m - 1) / (m + 1), with s and the leading term in two
// doubles (error-free transformations: Dekker 1971, Knuth) and the tail of the
// series, s^3 (1/3 + s^2/5 + ...), |s| < 0.1716, in one.  Error below 4e-18.
STX_HD void log_dd(double x, double &hi, double &lo) {
  long long b;
  double m;
  memcpy(&b, &x, sizeof b);
  int e = (int)(b >> 52) - 1023;
  b = (b & 0x000fffffffffffffll) | 0x3ff0000000000000ll;
  memcpy(&m, &b, sizeof m);
  if (m > 1.4142135623730951) { m = m * 0.5; e = e + 1; }
  const double u = m - 1.0, v = m + 1.0, vl = (m - (v - 1.0));
  const double rv = 1.0 / v;
  const double s = u * rv;
  const double sl = (fma(-s, v, u) - s * vl) * rv;
  const double z = s * s;
  double q = 1.0 / 23.0;
  q = fma(q, z, 1.0 / 21.0);
  q = fma(q, z, 1.0 / 19.0);
  q = fma(q, z, 1.0 / 17.0);
  q = fma(q, z, 1.0 / 15.0);
  q = fma(q, z, 1.0 / 13.0);
  q = fma(q, z, 1.0 / 11.0);
  q = fma(q, z, 1.0 / 9.0);
  q = fma(q, z, 1.0 / 7.0);
  q = fma(q, z, 1.0 / 5.0);
  q = fma(q, z, 1.0 / 3.0);
  const double tail = 2.0 * (s * z) * q;
  const double de = (double)e;
  const double A = de * LN2_HI, B = 2.0 * s;      // A is exact
  const double S = A + B, bb = S - A;
  const double err = (A - (S - bb)) + (B - bb);
  const double l = err + (fma(de, LN2_LO, 2.0 * sl) + tail);
  hi = S + l;
  lo = l - (hi - S);
}

// A T^b exp(nE rt), ln T = lh + ll: one exponential of b ln T + nE rt, whose
// argument is carried in two doubles, in the place of a power and an exponential.
// A power costs several times an exponential, and a right-hand side of the
// 9-species H2/air mechanism took 14 of them.  The argument's only rounding is
// nE rt's, which the separate exponential has too, so the result is no further
// from the exact one than theirs.
STX_HD double arrhenius_dd(double A, double b, double nE, double lh, double ll, double rt) {
  const double p = b * lh, q = nE * rt;
  const double s = p + q, bb = s - p;
  const double err = (p - (s - bb)) + (q - bb);
  const double e = err + fma(b, ll, fma(b, lh, -p));
  const double x = exp(s);
  return A * fma(x, e, x);
}
