// Pair terms and reductions shared by the real-space kernels.
#pragma once

#include "gb_internal.h"

namespace gb {

// FFParticle::CalcEn for lambda = 1 (src/FFParticle.cpp:295-325); the caller
// has checked r^2 < Rcut^2.  For n = 12 the (sigma^2/r^2)^6 term is the square
// of the attractive term instead of pow(), one rounding apart.
__device__ __forceinline__ double lj_energy(const FF &ff, double distSq,
                                            int idx) {
  double rRat2 = ff.sigmaSq[idx] / distSq;
  double rRat4 = rRat2 * rRat2;
  double attract = rRat4 * rRat2;
  double n = ff.nexp[idx];
  double repulse = (n == 12.0) ? attract * attract : pow(rRat2, n * 0.5);
  return ff.eps_cn[idx] * (repulse - attract);
}

// FFParticle::CalcVir for lambda = 1 (src/FFParticle.cpp:344-359)
__device__ __forceinline__ double lj_virial(const FF &ff, double distSq,
                                            int idx) {
  double rNeg2 = 1.0 / distSq;
  double rRat2 = rNeg2 * ff.sigmaSq[idx];
  double rRat4 = rRat2 * rRat2;
  double attract = rRat4 * rRat2;
  double n = ff.nexp[idx];
  double repulse = (n == 12.0) ? attract * attract : pow(rRat2, n * 0.5);
  return ff.eps_cn_6[idx] * (ff.nOver6[idx] * repulse - attract) * rNeg2;
}

// erfc(alpha r) / r from r^2 = s.  Inside the table's range: the segment
// from the bits of s (exponent and top 6 mantissa bits), u = 2 (s - a) / h
// - 1 in [-1, 1) exactly (a is s with the lower mantissa bits cleared, 2 / h
// a power of two), and a degree-8 polynomial in u (Chebyshev interpolant of
// the function on the segment, fitted on the host in extended precision;
// relative error near 1e-16 plus the FP64 rounding of the Horner steps).
// Outside it (r^2 < 0.5 A^2 or no table): the direct formula.  About a dozen
// FP64 operations against ~100 for sqrt, erfc and the division, which
// matters on GB300's two FP64 lanes per SM and clock.
// The segment polynomial of table `tab` at r^2 = s; false outside the range.
__device__ __forceinline__ bool seg_poly(const FF &ff, const double *tab,
                                         double s, double *out) {
  long long bits = __double_as_longlong(s);
  int seg = (int)(bits >> 46) - ff.etab_key0;
  if (tab == nullptr || (unsigned)seg >= (unsigned)ff.etab_nseg)
    return false;
  double a = __longlong_as_double(bits & ~((1LL << 46) - 1));
  double scale = __longlong_as_double((2053LL - (bits >> 52)) << 52);
  double u = fma(s - a, scale, -1.0);
  const double *c = tab + (size_t)seg * (ETAB_DEG + 1);
  double p = __ldg(c + ETAB_DEG);
#pragma unroll
  for (int m = ETAB_DEG - 1; m >= 0; --m)
    p = fma(p, u, __ldg(c + m));
  *out = p;
  return true;
}
__device__ __forceinline__ double erfc_over_r(const FF &ff, double s) {
  double p;
  if (seg_poly(ff, ff.erfc_tab, s, &p))
    return p;
  double r = sqrt(s);
  return erfc(ff.alpha * r) / r;
}

// FFParticle::CalcCoulomb, Ewald real-space term (src/FFParticle.cpp:361-399)
__device__ __forceinline__ double coulomb_energy(const FF &ff, double distSq,
                                                 double qq) {
  if (ff.rcutCoulSq < distSq)
    return 0.0;
  if (ff.ewald)
    return qq * erfc_over_r(ff, distSq);
  return qq / sqrt(distSq);
}

// FFParticle::CalcCoulombVir (src/FFParticle.cpp:401-446) by the formula; the
// pair walks take the Ewald force factor from pair_poly inside its range.
__device__ __forceinline__ double coulomb_virial(const FF &ff, double distSq,
                                                 double qq) {
  if (ff.rcutCoulSq < distSq)
    return 0.0;
  double dist = sqrt(distSq);
  if (ff.ewald) {
    double constValue = ff.alpha * M_2_SQRTPI;
    double expConstValue = exp(-1.0 * ff.alphaSq * distSq);
    double temp = 1.0 - erf(ff.alpha * dist);
    return qq * (temp / dist + constValue * expConstValue) / distSq;
  }
  return qq / (distSq * dist);
}

// ---- FP64 work moved to the integer and FP32 pipes ----
// GB300 retires two FP64 lanes per SM and clock, 64 times fewer than FP32 or
// integer ones; comparisons and conversions are FP64 instructions too.
__device__ __forceinline__ long long bits64(double v) {
  return __double_as_longlong(v);
}
__device__ __forceinline__ bool nonzero(double v) {
  return (bits64(v) << 1) != 0;
}
// a > b of two non-negative values (NaN above all), on the integer pipe
__device__ __forceinline__ bool gt_pos(double a, double b) {
  return bits64(a) > bits64(b);
}

// FP32 value of a positive FP64 number in FP32's normal range, truncated, and
// the exact FP64 value of a normal FP32 one, by moving bits: the conversion
// instructions run at the FP64 rate.
__device__ __forceinline__ float trunc_f32(double v) {
  return __uint_as_float((unsigned)(bits64(v) >> 29) - (896u << 23));
}
__device__ __forceinline__ double widen_f64(float f) {
  const unsigned b = __float_as_uint(f);
  const unsigned hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20));
  return __hiloint2double((int)hi, (int)(b << 29));
}

// 1 / s, s positive and well inside FP32's range, by one step of Householder's
// third-order iteration y (1 + e + e^2), e = 1 - s y, from the FP32 reciprocal of
// s truncated to FP32 (|e| < 2^-22): e^3 is below 2^-66, so that what is left is
// the rounding of the last step, half a unit of the last place (as measured over
// 2 million s against 113 bits, and as two Newton steps and a division leave).
__device__ __forceinline__ double recip_cubic(double s) {
  const double y = widen_f64(__frcp_rn(trunc_f32(s)));
  const double e = fma(-s, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// a / s with the product's own rounding corrected by its residual: to the last
// bit, y = recip_cubic(s)
__device__ __forceinline__ double quot_pos(double a, double s, double y) {
  const double q = a * y;
  return fma(fma(-q, s, a), y, q);
}
// these and the bit conversions hold for 2^-60 < s < 2^60
__device__ __forceinline__ bool in_fast_range(double s) {
  const int e = __double2hiint(s) >> 20;
  return e > 1023 - 60 && e < 1023 + 60;
}

// A segment polynomial of ff.pair_tab at the position u in [-1, 1) that the
// bits b of r^2 give: degrees 0-6 in FP64, 7 and 8 (the halves of c6.y) in FP32.
// Those two add less than 1e-11 of the value for alpha r up to 3.4 (a tolerance of
// 1e-5; 1.2e-9 up to 4.8, 1e-10), so their rounding is below 2^-60 (2^-53) of it:
// against 113 bits over r from 0.7 A to Rcut the largest and the rms error are
// those of nine FP64 degrees to four digits (2.2e-16 and 6.6e-17; 2.8e-16 and
// 7.1e-17 at 1e-10).  With degree 6 in FP32 too the largest was 5.6e-16 at 1e-10.
__device__ __forceinline__ double pair_poly_at(long long b, double2 c01,
                                               double2 c23, double2 c45,
                                               double2 c6) {
  const double u = fma(
      2.0, __longlong_as_double(((b << 6) & 0x000fffffffffffffLL) |
                                0x3ff0000000000000LL), -3.0);
  const float uf = fmaf(
      2.0f, __int_as_float(((int)(b >> 23) & 0x007fffff) | 0x3f800000), -3.0f);
  const long long f = bits64(c6.y);
  const float t = fmaf(__int_as_float((int)(f >> 32)), uf, __int_as_float((int)f));
  double p = fma(widen_f64(t), u, c6.x);
  p = fma(p, u, c45.y);
  p = fma(p, u, c45.x);
  p = fma(p, u, c23.y);
  p = fma(p, u, c23.x);
  p = fma(p, u, c01.y);
  return fma(p, u, c01.x);
}

// Segment polynomial `which` (0 energy, 1 force factor) of ff.pair_tab at
// s; false outside its range.  The segment and the position u in [-1, 1) in
// it come from the bits of s, as in seg_poly.
__device__ __forceinline__ bool pair_poly(const FF &ff, int which, double s,
                                          double *out) {
  const long long b = bits64(s);
  const int seg = (int)(b >> 46) - ff.etab_key0;
  if (ff.pair_tab == nullptr || (unsigned)seg >= (unsigned)ff.etab_nseg)
    return false;
  const double2 *c = (const double2 *)(ff.pair_tab + ((size_t)seg * 2 + which) * 8);
  *out = pair_poly_at(b, __ldg(c), __ldg(c + 1), __ldg(c + 2),
                      __ldg(c + 3));
  return true;
}
// Soft-core squared distance at coupling lambda (src/FFParticle.cpp:301-308):
// cbrt(sc_alpha (1 - lambda)^sc_power max(sigma^6, sc_sigma^6) + r^6).
__device__ __forceinline__ double soft_rsq(const FF &ff, double distSq,
                                           int idx, double lambda) {
  double sigma6 = ff.sigmaSq[idx] * ff.sigmaSq[idx] * ff.sigmaSq[idx];
  sigma6 = fmax(sigma6, ff.sc_sigma_6);
  double dist6 = __dmul_rn(__dmul_rn(distSq, distSq), distSq);
  double lambdaCoef = ff.sc_alpha * pow((1.0 - lambda), (double)ff.sc_power);
  double softDist6 = __dadd_rn(__dmul_rn(lambdaCoef, sigma6), dist6);
  return cbrt(softDist6);
}

// FFParticle::CalcEn at coupling lambda (src/FFParticle.cpp:295-316); the
// caller has checked r^2 < Rcut^2.
__device__ __forceinline__ double lj_energy_lambda(const FF &ff, double distSq,
                                                   int idx, double lambda) {
  if (lambda >= 0.999999)
    return lj_energy(ff, distSq, idx);
  return lambda * lj_energy(ff, soft_rsq(ff, distSq, idx, lambda), idx);
}

// FFParticle::CalcCoulomb at coupling lambda (src/FFParticle.cpp:361-387):
// the soft-core distance only with sc_coul.
__device__ __forceinline__ double coulomb_energy_lambda(const FF &ff,
                                                        double distSq, int idx,
                                                        double qq,
                                                        double lambda) {
  if (ff.rcutCoulSq < distSq)
    return 0.0;
  if (lambda >= 0.999999)
    return coulomb_energy(ff, distSq, qq);
  double r2 = ff.sc_coul ? soft_rsq(ff, distSq, idx, lambda) : distSq;
  double dist = sqrt(r2);
  double e = ff.ewald ? qq * erfc(ff.alpha * dist) / dist : qq / dist;
  return lambda * e;
}

// Sums over a warp of four values with six additions a lane instead of
// twenty: the lanes share the values out as the sums fold.  Lane 0 has v[0],
// lane 8 v[1], lane 16 v[2], lane 24 v[3].
__device__ __forceinline__ double warp_sum4(const double (&v)[4]) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, g = lane & 8;
  double a = h ? v[2] : v[0], b = h ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
  b += __shfl_xor_sync(0xffffffffu, h ? v[1] : v[3], 16);
  double c = g ? b : a;
  c += __shfl_xor_sync(0xffffffffu, g ? a : b, 8);
  for (int o = 4; o > 0; o >>= 1)
    c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;
}
// Two values, five additions: lane 0 has x, lane 16 y.
__device__ __forceinline__ double warp_sum2(double x, double y) {
  const bool h = threadIdx.x & 16;
  double a = (h ? y : x) + __shfl_xor_sync(0xffffffffu, h ? x : y, 16);
  for (int o = 8; o > 0; o >>= 1)
    a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// The last CTA of the grid to get here (every thread of every CTA calls):
// true in that CTA, where the others' writes before the call can be read.
// The ticket counts back to zero by itself.
__device__ __forceinline__ bool last_cta(unsigned *ticket) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  return last != 0;
}

// Block-wide sum of one double, deterministic order; result valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh) {
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_down_sync(0xffffffffu, v, o);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0)
    sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NT / 32; ++i)
      r += sh[i];
  }
  __syncthreads();
  return r;
}

}  // namespace gb
