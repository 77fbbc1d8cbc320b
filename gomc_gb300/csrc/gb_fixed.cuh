// Phases in 62-bit fixed point: exact fractions of a turn and their cosine and
// sine by integer arithmetic, which GB300 retires 32 to 64 times faster than
// FP64, with errors below 2^-58.
#pragma once

namespace gb {

// ---- 62-bit fixed point ----
// a b 2^-62, rounded
__device__ __forceinline__ long long mulq62(long long a, long long b) {
  const long long hi = __mul64hi(a, b);
  const unsigned long long lo = (unsigned long long)a * (unsigned long long)b;
  return (long long)(((unsigned long long)hi << 2) | (lo >> 62)) +
         (long long)((lo >> 61) & 1);
}

// x / L as a 64-bit fraction of a turn: the FP64 quotient and, from the exact
// remainder, what it misses
__device__ __forceinline__ unsigned long long turn64(double x, double L) {
  const double t = x / L;
  const double lo = fma(-t, L, x) / L;
  return __double2ull_rn((t - floor(t)) * 18446744073709551616.0) +
         (unsigned long long)__double2ll_rn(lo * 18446744073709551616.0);
}

struct Cis {
  long long c, s;  // cos and sin times 2^62
};

// exp(2 pi i u / 2^64): quarter turn by integer arithmetic, then the Taylor
// series on |x| <= pi/4 to x^19 and x^20 (truncation below 2^-65).
__device__ inline Cis cis_q62(unsigned long long u) {
  const long long s = (long long)u;
  const long long q = (long long)((unsigned long long)s + (1ull << 61)) >> 62;
  const long long r = (long long)(u - ((unsigned long long)q << 62));
  // x = r 2 pi / 2^64 in 2^-62: r (pi / 2), pi/2 in 2^-62
  const long long x = mulq62(r, 7244019458077122842LL);
  const long long x2 = mulq62(x, x);
  // 1/k! in 2^-62 (integer division: exact to the last bit)
  constexpr long long ONE = 1LL << 62;
  long long ps = -(ONE / 121645100408832000LL);         // -1/19!
  ps = ONE / 355687428096000LL + mulq62(x2, ps);        //  1/17!
  ps = -(ONE / 1307674368000LL) + mulq62(x2, ps);
  ps = ONE / 6227020800LL + mulq62(x2, ps);
  ps = -(ONE / 39916800LL) + mulq62(x2, ps);
  ps = ONE / 362880LL + mulq62(x2, ps);
  ps = -(ONE / 5040LL) + mulq62(x2, ps);
  ps = ONE / 120LL + mulq62(x2, ps);
  ps = -(ONE / 6LL) + mulq62(x2, ps);
  const long long sn = x + mulq62(mulq62(x, x2), ps);
  long long pc = ONE / 2432902008176640000LL;           //  1/20!
  pc = -(ONE / 6402373705728000LL) + mulq62(x2, pc);
  pc = ONE / 20922789888000LL + mulq62(x2, pc);
  pc = -(ONE / 87178291200LL) + mulq62(x2, pc);
  pc = ONE / 479001600LL + mulq62(x2, pc);
  pc = -(ONE / 3628800LL) + mulq62(x2, pc);
  pc = ONE / 40320LL + mulq62(x2, pc);
  pc = -(ONE / 720LL) + mulq62(x2, pc);
  pc = ONE / 24LL + mulq62(x2, pc);
  pc = -(ONE / 2LL) + mulq62(x2, pc);
  const long long cs = ONE + mulq62(x2, pc);
  switch ((int)q & 3) {
    case 0: return {cs, sn};
    case 1: return {-sn, cs};
    case 2: return {-cs, -sn};
    default: return {sn, -cs};
  }
}

__device__ __forceinline__ Cis cis_mul(Cis a, Cis b) {
  return {mulq62(a.c, b.c) - mulq62(a.s, b.s),
          mulq62(a.c, b.s) + mulq62(a.s, b.c)};
}

}  // namespace gb
