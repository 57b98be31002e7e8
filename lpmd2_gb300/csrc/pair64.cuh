// pair64.cuh -- FP64 pair arithmetic for GB300's FP64 unit (2 lanes a clock and SM): as few FP64
// instructions a pair as the result needs, decisions on the integer and FP32 pipes.  Shared by the
// FP64 passes (force64.cuh) and the direct entry point (static_forces.cu).
#pragma once

#include "potentials.cuh"

namespace gbmd {

// An FP32 value within one unit in the last place of the double, by truncation on the integer pipe
// (a conversion would run on the FP64 unit).  Values below the FP32 normal range give 0, values
// above it an infinity.
__device__ __forceinline__ float trunc32(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int e = (int)((hi >> 20) & 0x7ffu) - 896;
  unsigned m = (hi << 3) | (lo >> 29);
  m = ((unsigned)e << 23) | (m & 0x7fffffu);
  if (e <= 0) m = 0u;
  if (e >= 255) m = 0x7f800000u;
  return __uint_as_float(m | (hi & 0x80000000u));
}

// Whether ref_wrap wraps d, decided on the bit patterns (its branches are d >= L/2 and d < -L/2);
// lhb: the bits of L/2.
__device__ __forceinline__ bool wraps_bits(double d, long long lhb) {
  const long long b = __double_as_longlong(d);
  const long long m = b & 0x7fffffffffffffffll;
  return b < 0 ? m > lhb : m >= lhb;
}

// Whether v is infinite or NaN, on the bit pattern.
__device__ __forceinline__ bool not_finite_bits(double v) {
  return ((unsigned)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u;
}

// 1 / x for x >= 0 by one step of Halley's iteration, y (1 + e + e^2) with e = 1 - x y, from the
// hardware's approximation (relative error below 2^-20, so e^3 is below the last bit).  1 / 0 is
// infinite, as with a division: the step alone would give a NaN.
__device__ __forceinline__ double rcp64(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  const double r = fma(y, fma(e, e, e), y);
  return not_finite_bits(y) ? y : r;
}

// 1 / sqrt(x) for x >= 0 by the third-order step of the same family (Householder's iteration; the
// binomial series of (1 - e)^(-1/2)): y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2.  1 / sqrt(0) is infinite.
__device__ __forceinline__ double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  const double r = fma(y * e, fma(0.375, e, 0.5), y);
  return not_finite_bits(y) ? y : r;
}

// sqrt(x) from x and rsqrt64(x); 0 for 0.
__device__ __forceinline__ double sqrt64(double x, double ir) { return not_finite_bits(ir) ? x : x * ir; }

// Lower bound of one axis of the reference's displacement (one wrap) from truncated coordinates: each
// is off by at most one unit in the last place, so a component is below its truth by at most tol
// (the wrap may pick the other image only where both are half a box long, within tol).
__device__ __forceinline__ float axis_bound(float a, float b, float L) {
  float d = fabsf(b - a);
  const float tol = 4.8e-7f * (fabsf(a) + fabsf(b) + L);
  if (d >= 0.5f * L) d = fabsf(d - L);
  return fmaxf(d - tol, 0.0f);
}

// Constants of a potential as the pair loops use them, computed on the host (kernel arguments: the
// FP64 instructions read them from the constant bank).
struct Pair64 {
  double c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0;
  double phi = 1.0;  // prefactor of the many-body force, folded into the stored embedding factor
};

inline Pair64 pair64_constants(const PotParams& P) {
  Pair64 c;
  const double* p = P.p;
  if (P.kind == POT_LJ) {
    c.c0 = p[0] * p[0];      // sigma^2
    c.c1 = -48.0 * p[1];
    c.c2 = 24.0 * p[1];
    c.c3 = 4.0 * p[1];
  } else if (P.kind == POT_SC) {
    c.c0 = p[0] * P.an;                                  // e a^n
    c.c1 = -p[2] * p[0] * P.an;                          // -n e a^n
    c.phi = 0.5 * p[3] * p[4] * p[0] * P.am;             // m c e a^m / 2
  } else if (P.kind == POT_FS) {
    c.c0 = p[4] / p[6];          // B / d
    c.c1 = 3.0 * p[4] / p[6];
    c.phi = -0.5 * p[3];         // -A / 2
    c.c3 = 2.0 * p[2];           // 2 c2
  } else if (P.kind == POT_FSEXT) {
    c.c0 = p[6] * p[6];          // B^2
    c.c1 = 4.0 * p[6] * p[6];
    c.phi = -0.5 * p[5];
    c.c3 = 2.0 * p[2];
  } else if (P.kind == POT_GUPTA) {
    c.c0 = -p[2] / p[1];         // -p / r0
    c.c1 = -2.0 * p[4] / p[1];   // -2 q / r0
    c.c2 = -p[0] * p[2] / p[1];  // -A p / r0
    c.phi = p[3] * p[4] / p[1];  // B q / r0
  }
  return c;
}

// Lennard-Jones: g with F_i = g r_ij (r_ij = x_j - x_i); the pair's energy is added to ep if `count`.
__device__ __forceinline__ double lj_body64(const Pair64& c, double r2, bool count, double& ep) {
  const double inv = rcp64(r2);
  const double x = c.c0 * inv;
  const double r6 = x * x * x;
  if (count) ep = fma(r6, fma(c.c3, r6, -c.c3), ep);
  return (inv * r6) * fma(c.c1, r6, c.c2);
}

// Sum over the lanes of an atom of three components: after the first two exchanges every lane
// carries one of them (4 additions for 8 lanes instead of 9).  Lane `sub` returns component
// (sub / (lanes/4)) % 4 in exchange order: 0 x, 1 y, 2 z, 3 nothing.
__device__ __forceinline__ double atom_sum3(double x, double y, double z, int sub, int lanes) {
  const int h = lanes >> 1, q = lanes >> 2;
  const bool up = (sub & h) != 0, odd = (sub & q) != 0;
  double a = up ? z : x, b = up ? 0.0 : y;
  const double sa = up ? x : z, sb = up ? y : 0.0;
  a += __shfl_xor_sync(0xffffffffu, sa, h);
  b += __shfl_xor_sync(0xffffffffu, sb, h);
  double c = odd ? b : a;
  c += __shfl_xor_sync(0xffffffffu, odd ? a : b, q);
  for (int m = q >> 1; m > 0; m >>= 1) c += __shfl_xor_sync(0xffffffffu, c, m);
  return c;
}

}  // namespace gbmd
