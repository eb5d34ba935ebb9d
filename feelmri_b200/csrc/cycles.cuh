// exp(i 2 pi c) of a phase c in cycles.
#pragma once
#include <cstdint>

namespace fm {

// Two FP32 values in one 64-bit register and the packed FP32 instructions.
using f32x2 = unsigned long long;
__device__ inline f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ inline void unpack2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ inline f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ inline f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// A phase outside [-2^19, 2^19] cycles, or one that is not a number.
__device__ __noinline__ void cis_far(double c, float &re, float &im) {
  float s;
  sincospif(2.f * (float)(c - rint(c)), &s, &re);
  im = s;
}

// exp(i 2 pi c) of two phases in FP32: (re0, re1), (im0, im1), and -(im0, im1).
//
// c + 1.5 2^20 is a double whose low word is c modulo one cycle in steps of
// 2^-32 cycles, so the reduction is one addition and the error it leaves is
// 1e-9 rad.  The fraction, less half a cycle where that brings it within a
// quarter of 0, becomes y in [-1, 1] quarter cycles; sin and cos of pi/2 y are
// polynomials in y^2 fitted to least maximum error by Lawson's iteratively
// reweighted least squares on Chebyshev points, each coefficient rounded to
// FP32 before the next were fitted (largest error 1.4e-7 and 9e-8, rms 2.6e-8
// and 2.3e-8 including rounding; tests/test_gpu_signal_units.py).  About 36
// instructions a pair, where sincosf takes some 80.
__device__ inline void cis_cycles2(double c0, double c1, f32x2 &re, f32x2 &im, f32x2 &neg_im) {
  const double t0 = c0 + 0x1.8p20, t1 = c1 + 0x1.8p20;
  const uint32_t u0 = (uint32_t)__double2loint(t0), u1 = (uint32_t)__double2loint(t1);
  const uint32_t h0 = u0 + 0x40000000u, h1 = u1 + 0x40000000u;
  const uint32_t m = 0x80000000u;
  const float y0 = (float)(int32_t)(u0 ^ (h0 & m)), y1 = (float)(int32_t)(u1 ^ (h1 & m));
  const f32x2 y = mul2(pack2(y0, y1), pack2(0x1p-30f, 0x1p-30f));
  const f32x2 z = mul2(y, y);
#define FM_C2(x) pack2(x, x)
  f32x2 s = fma2(z, FM_C2(0x1.3911b2p-13f), FM_C2(-0x1.31fbeep-8f));
  f32x2 c = fma2(z, FM_C2(-2.3402006263495423e-05f), FM_C2(0.0009167332900688052f));
  s = fma2(s, z, FM_C2(0x1.466504p-4f));
  c = fma2(c, z, FM_C2(-0.020861899480223656f));
  s = fma2(s, z, FM_C2(-0x1.4abba2p-1f));
  c = fma2(c, z, FM_C2(0.2536690831184387f));
  s = fma2(s, z, FM_C2(0x1.921fb4p+0f));
  c = fma2(c, z, FM_C2(-1.2337005138397217f));
  s = mul2(s, y);
  c = fma2(c, z, FM_C2(1.f));
#undef FM_C2
  float s0, s1, r0, r1;
  unpack2(s, s0, s1);
  unpack2(c, r0, r1);
  const uint32_t g0 = h0 & m, g1 = h1 & m;
  float i0 = __uint_as_float(__float_as_uint(s0) ^ g0), i1 = __uint_as_float(__float_as_uint(s1) ^ g1);
  r0 = __uint_as_float(__float_as_uint(r0) ^ g0);
  r1 = __uint_as_float(__float_as_uint(r1) ^ g1);
  // the sum kept its exponent: both phases were in range
  if ((((uint32_t)__double2hiint(t0) ^ 0x41300000u) | ((uint32_t)__double2hiint(t1) ^ 0x41300000u)) >> 20) {
    cis_far(c0, r0, i0);
    cis_far(c1, r1, i1);
  }
  re = pack2(r0, r1);
  im = pack2(i0, i1);
  neg_im = im ^ 0x8000000080000000ull;
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
