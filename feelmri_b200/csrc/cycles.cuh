// exp(i 2 pi c) of a phase c in cycles.
#pragma once
#include <cstdint>

namespace fm {

// exp(i 2 pi c) in FP32.
//
// c + 1.5 2^20 is a double whose low word is c modulo one cycle in steps of
// 2^-32 cycles, so the reduction is one addition and the error it leaves is
// 1e-9 rad; a phase beyond 2^19 cycles is reduced first.  The fraction, less
// half a cycle where that brings it within a quarter of 0, becomes y in [-1, 1]
// quarter cycles; sin and cos of pi/2 y are polynomials in y^2 fitted to least
// maximum error by Lawson's iteratively reweighted least squares on Chebyshev
// points, each coefficient rounded to FP32 before the next were fitted (largest
// error 1.4e-7 and 9e-8, rms 2.6e-8 and 2.3e-8 including rounding).  About 20
// instructions, where sincosf takes some 40.
__device__ inline void cis_cycles(double c, float &re, float &im) {
  double t = c + 0x1.8p20;
  float scale = 0x1p-30f;
  if (((uint32_t)__double2hiint(t) ^ 0x41300000u) >> 20) {  // the sum's exponent changed: c is out of range
    c -= rint(c);
    t = c + 0x1.8p20;
    if (c != c) scale = (float)c;
  }
  const uint32_t u = (uint32_t)__double2loint(t), h = u + 0x40000000u, half = h & 0x80000000u;
  const float y = (float)(int32_t)(u ^ half) * scale, z = y * y;
  float s = fmaf(z, 0x1.3911b2p-13f, -0x1.31fbeep-8f);
  float k = fmaf(z, -2.3402006263495423e-05f, 0.0009167332900688052f);
  s = fmaf(s, z, 0x1.466504p-4f);
  k = fmaf(k, z, -0.020861899480223656f);
  s = fmaf(s, z, -0x1.4abba2p-1f);
  k = fmaf(k, z, 0.2536690831184387f);
  s = fmaf(s, z, 0x1.921fb4p+0f);
  k = fmaf(k, z, -1.2337005138397217f);
  s = s * y;
  k = fmaf(k, z, 1.f);
  im = __uint_as_float(__float_as_uint(s) ^ half);
  re = __uint_as_float(__float_as_uint(k) ^ half);
}

// 1 / 2 pi and float(pi) / pi to twice FP64 precision.
constexpr double kInv2Pi = 0x1.45f306dc9c883p-3, kInv2PiLo = -0x1.6b01ec5417056p-57;
constexpr double kPiRatio = 0x1.0000007784b2dp+0, kPiRatioLo = -0x1.c235d1ac21643p-57;

// A phase in FP64 as a sum of products, reduced exactly: `f` whole cycles
// dropped, `e` what rounding left out.
struct Cycles {
  double f = 0.0, e = 0.0;
  // adds (hi + lo) * x
  __device__ void add(double hi, double lo, double x) {
    const double p = hi * x;
    e += fma(hi, x, -p) + lo * x;
    f += p - rint(p);
    f -= rint(f);
  }
  // adds x t / 2 pi
  __device__ void add_turn(double x, double t) {
    const double p = x * t;
    add(p, 0.0, kInv2Pi);
    e += fma(x, t, -p) * kInv2Pi + p * kInv2PiLo;
  }
  __device__ void cis(double &re, double &im) const { sincospi(2.0 * (f + e), &im, &re); }
};

}  // namespace fm
