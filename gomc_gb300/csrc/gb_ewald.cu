// The box-wide Ewald sums as matrix products on the tensor cores, with more
// than FP64's accuracy.
//
//   structure factor  S(k) = sum_j q_j exp(i k . r_j)
//                     (Ewald::BoxReciprocalSetup/Sums, src/Ewald.cpp:193-361)
//   reciprocal force  F_a = 2 q_a sum_k prefact_k (sin(k.r_a) S_R
//                     - cos(k.r_a) S_I) k  (Ewald::BoxForceReciprocal,
//                     src/Ewald.cpp:1496-1596)
//
// exp(i k . r) is a product over the axes, so with the four real y-z products
// Y(p) = {cos cos, cos sin, sin cos, sin sin} of each pair p = (|n_y|, |n_z|)
// and X(n) = {cos, sin}(n_x t_x),
//   sums    D[4p + c, 2n + s] = sum_atoms Y_c(p, atom) q X_s(n, atom),
//           from which four k-vectors (the signs of n_y, n_z) take their sums;
//   forces  D_w[atom, 2n + s] = sum_pairs Y_c(p, atom) C_w[4p + c, 2n + s],
//           C_w the structure factors times prefactor and k_w, folded over
//           the four signs; the atom then sums D_w over n with its own X.
// Both are contractions of two multiply-adds per atom and k-vector and
// component.  On the FP64 pipe (two lanes per SM and clock) they cannot run
// below 2 ms / 6 ms on 8,000 waters; FP32 pairs would cost accuracy.  Instead
// both factors are 55-bit fixed-point numbers cut into seven signed 8-bit
// digits, held exactly in FP16 (the scheme of Ozaki, Ogita, Oishi and Rump,
// Numer. Algorithms 59 (2012) 95, with digits of a fixed scale): a product of
// digit i and digit j is exact, and sums over 128 terms of the digit pairs with
// i + j = d stay below 2^24 and are exact in the FP32 accumulators of d = 0..6.
// Pairs with i + j >= 7 are left out: with the rounding of the factors a term is
// within 2^-51 of the unit (the power of two above the largest charge of its
// class, or above a column's largest C), some 2^-54 rms, and the errors of n terms
// add up as sqrt(n).  Measured against sums of exact phases, in units of the sums'
// rms: 3.8e-16 (256 waters), 5.5e-16 (8,000), 8.3e-16 (20,000), where an FP64
// recurrence had 2.3e-15, 1.0e-14 and 1.3e-14.  The seven accumulators sit side by
// side in tensor memory; every 128 terms the CTA adds them into one 64-bit integer
// per output.  Integer sums do not depend on their order, so chunks of atoms are
// added by 64-bit integer atomics and results are equal run to run.
//
// A CTA has 128 rows of D and up to 64 columns, one CTA per SM (two stages of
// 32 terms of Y and three of the other operand in shared memory).  Sixteen
// warps form the Y operand of the next stage -- one 64 x 64-bit fixed-point
// product per element, cut into digits by byte permutes -- while the tensor
// core works on the last one; a seventeenth starts the products.  The other operand (X or C) is cut
// beforehand and copied asynchronously by three more, a stage ahead (16-byte
// copies: only the columns in use are copied, and bulk copies of that many
// pieces took 75 cycles each to start).  The slices of that operand lie side by
// side as columns, so digit i of Y meets several digits of it in one product.
// Products started one after another run in that order only where their
// accumulator and shape are the same, so the accumulators form two or three
// blocks and every product writes one whole block: digit i of Y meets slices
// d - i, those below 0 being zeros ahead of the operand's own (18 or 24 products
// a stage instead of 56, a third or a fifth of their columns zeros).
// Forming Y on the fly keeps its 7 x 2 bytes per element out of memory.  Pairs
// are sorted by their largest n_x, so the columns beyond the k-sphere are
// skipped (a third of the product).
// Measured on 8,000 waters (24,658 k-vectors), per launch: sums 141 us, forces
// 429 us (the FP64 kernels before: 11 ms and 12.1 ms); sums of 20,000 waters
// 692 us.  A stage takes some 3,900 cycles: its products read 193 KB of shared
// memory (1,510 cycles) and keep the tensor pipe 39-42 % busy; the warps that form
// Y and add the windows issue 56 % of the cycles, the rest is their load latency.
//
// Phases: u = (x / L) 2^64 is a fraction of a turn to 2^-64, n u is exact
// integer arithmetic, and cos and sin come from their Taylor series in 62-bit
// fixed point: the error does not grow with n as in an FP64 recurrence.
#include "gb_box.h"
#include "gb_fixed.cuh"
#include "gb_pair.cuh"

#include <cuda_fp16.h>

#include <cmath>

namespace gb {

namespace {

constexpr int TM = 128;      // rows of D per CTA
constexpr int TK = 32;       // terms per stage
constexpr int NSL = 7;       // digits per operand
constexpr int WIN = 4;       // stages per exact window: 128 terms
constexpr int ET = 512;      // threads that form the left operand
constexpr int CW = 3;        // warps that copy the right operand
constexpr int CTA = ET + 32 + 32 * CW;
constexpr int NT_MAX = 64;   // columns per CTA: 7 x 64 of 512 TMEM columns
// slices of zeros ahead of the right operand's with n columns a slice (product
// below), and the rows of 8 terms of all of them where a tile has nt columns
__host__ __device__ constexpr int zeros(int n) { return n <= 48 ? 4 : 2; }
__host__ __device__ constexpr int ring_rows(int nt) {
  return (zeros(nt) + NSL) * nt;  // 64 columns: more than 48 of its columns take
}
constexpr int A_KO = TM * 16 + 32;              // bytes between 8-term groups
constexpr int A_SLICE = TK / 8 * A_KO;          // bytes
constexpr int A_STAGE = NSL * A_SLICE;

// 2^-62 value as (hi, lo) with a signed low half, v = hi 2^32 + lo: a product
// then takes three 32 x 32-bit multiplies
__device__ __forceinline__ int2 balance(long long v) {
  const int lo = (int)v;
  return make_int2((int)((v - lo) >> 32), lo);
}

// 128 in each of the seven digit bytes: with it added, byte j holds the
// balanced digit j plus 128
constexpr unsigned long long DIGIT_BIAS = 0x0080808080808080ull;

// Biased digits (56 bits) of a 2^-62 value rounded to 2^-54
__device__ __forceinline__ unsigned long long digits_q62(long long v) {
  return (unsigned long long)((v + 128) >> 8) + DIGIT_BIAS;
}
// digit byte -> FP16: 1024 + byte is the pattern 0x6400 | byte
__device__ __forceinline__ __half digit_half(unsigned long long w, int j) {
  const unsigned short h = (unsigned short)(0x6400u | ((w >> (8 * j)) & 0xffu));
  return __hsub(__ushort_as_half(h), __ushort_as_half(0x6480));  // - 1152
}
__device__ __forceinline__ unsigned digit_pair(unsigned h) {
  const __half2 v = __hsub2(*reinterpret_cast<__half2 *>(&h),
                            __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<const unsigned *>(&v);
}

// Seven slices (slice 0 the leading digit) of eight elements given as biased
// digits, each slice as 16 bytes at dst + slice * stride.
__device__ __forceinline__ void store_slices(const unsigned long long (&w)[8],
                                             unsigned char *dst, int stride) {
  unsigned o[NSL][4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const unsigned al = (unsigned)w[2 * t], bl = (unsigned)w[2 * t + 1];
    const unsigned ah = (unsigned)(w[2 * t] >> 32) | 0x64000000u,
                   bh = (unsigned)(w[2 * t + 1] >> 32) | 0x64000000u;
    constexpr unsigned C = 0x64646464u;
    const unsigned x01 = __byte_perm(al, bl, 0x5140);
    const unsigned x23 = __byte_perm(al, bl, 0x7362);
    o[6][t] = digit_pair(__byte_perm(x01, C, 0x4140));
    o[5][t] = digit_pair(__byte_perm(x01, C, 0x4342));
    o[4][t] = digit_pair(__byte_perm(x23, C, 0x4140));
    o[3][t] = digit_pair(__byte_perm(x23, C, 0x4342));
    o[2][t] = digit_pair(__byte_perm(ah, bh, 0x7430));
    o[1][t] = digit_pair(__byte_perm(ah, bh, 0x7531));
    o[0][t] = digit_pair(__byte_perm(ah, bh, 0x7632));
  }
#pragma unroll
  for (int s = 0; s < NSL; ++s)
    *reinterpret_cast<uint4 *>(dst + s * stride) =
        make_uint4(o[s][0], o[s][1], o[s][2], o[s][3]);
}

// Biased digits of the product of two balanced 2^-62 values, to 2^-54
__device__ __forceinline__ unsigned long long product_digits(int2 a, int2 b) {
  long long t = (long long)a.x * b.y;
  t += (long long)a.y * b.x;
  long long p = (long long)a.x * b.x +
                (long long)((DIGIT_BIAS << 6) + 32ull);  // 2^-60
  p += t >> 32;
  return (unsigned long long)p >> 6;
}

// ---- mbarrier, bulk copy, tcgen05 ----
__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// Wait of at most `limit` polls for a phase, the first of them immediate, the
// others suspended for a time; false when it gives up, or when another warp has
// (*bad).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity,
                                          const int *bad, unsigned limit) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  for (unsigned it = 1; !ok && it < limit; ++it) {
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (bad && (it & 63u) == 63u && *(volatile const int *)bad)
      break;
  }
  return ok;
}
// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void copy16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src)
               : "memory");
}
// K-major operand without swizzle: 8 x 16-byte core matrices, `lbo` bytes
// between the 8-term groups, 128 between the 8-row groups.
__device__ __forceinline__ uint64_t smem_desc(unsigned addr, unsigned lbo) {
  return (uint64_t)((addr >> 4) & 0x3fff) | (uint64_t)(lbo >> 4) << 16 |
         (uint64_t)(128 >> 4) << 32 | 1ull << 46;
}
// One product, started by the lane with `lead` set (the whole warp calls: code
// without a divergent branch keeps the descriptors in uniform registers; a
// product started from a one-lane branch took about 170 cycles to issue).
__device__ __forceinline__ void mma_f16(unsigned lead, unsigned d, uint64_t a,
                                        uint64_t b, unsigned idesc, bool add) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"((unsigned)add), "r"(lead)
      : "memory");
}
// The products of 16 terms: digit i of Y on the slices from `b` on (digit 0's
// follows the zeros), `len` of them, into the accumulators d0 .. d0 + len - 1, for
// d0 + len > i; digits ascending.  The blocks are as few as 256 columns a product
// and the shared memory for the zeros allow: what a stage takes goes with the
// number of products more than with their width.  Forces of 8,000 waters (48
// columns): two blocks, 9 products of 39 slices' width, 1,616 us; 12 of 34, 1,672;
// 16 of 31, 1,744; seven blocks, 28 of 28, 2,053.
struct Product {
  int i, d0, len, b;
};
constexpr Product product(int n, int k) {
  const int wide[2] = {0, 2}, three[3] = {0, 1, 4};
  const int blocks = n <= 48 ? 2 : 3;
  for (int i = 0; i < NSL; ++i)
    for (int g = 0; g < blocks; ++g) {
      const int d0 = n <= 48 ? wide[g] : three[g];
      const int end = g + 1 == blocks ? NSL : n <= 48 ? wide[g + 1] : three[g + 1];
      if (i < end && k-- == 0)
        return {i, d0, end - d0, zeros(n) + d0 - i};
    }
  return {0, 0, 0, 0};
}
constexpr int products(int n) {
  int k = 0;
  while (product(n, k).len)
    ++k;
  return k;
}
// Products that share a column have the same accumulator and shape; the first of
// each block (which overwrites it) comes before the others; every i + j < NSL
// is in exactly one; and none leaves the operand's slices or 256 columns.
constexpr bool products_ordered(int n) {
  int met[NSL][NSL] = {};
  for (int k = 0; k < products(n); ++k) {
    const Product p = product(n, k);
    if (p.len * n > 256 || p.b < 0 || p.b + p.len > zeros(n) + NSL)
      return false;
    for (int m = 0; m < k; ++m) {
      const Product o = product(n, m);
      const bool share = o.d0 < p.d0 + p.len && p.d0 < o.d0 + o.len;
      if (share && (o.d0 != p.d0 || o.len != p.len || o.i >= p.i))
        return false;
    }
    for (int d = p.d0; d < p.d0 + p.len; ++d) {
      const int j = p.b + d - p.d0 - zeros(n);
      if (j >= 0 && (p.i + j != d || ++met[p.i][j] > 1))
        return false;
    }
  }
  for (int i = 0; i < NSL; ++i)
    for (int j = 0; i + j < NSL; ++j)
      if (!met[i][j])
        return false;
  return true;
}
static_assert(products_ordered(16) && products_ordered(32) &&
                  products_ordered(48) && products_ordered(64) && NT_MAX == 64,
              "products of one accumulator out of order");

// All products of a stage with N columns a slice.
template <int N>
__device__ __forceinline__ void mma_stage(unsigned lead, unsigned tmem,
                                          unsigned sa, unsigned sb, bool open) {
  constexpr int B_ROWS = (zeros(N) + NSL) * N;
  const uint64_t da = smem_desc(sa, A_KO), db = smem_desc(sb, B_ROWS * 16);
#pragma unroll
  for (int ks = 0; ks < TK / 16; ++ks)
#pragma unroll
    for (int k = 0; k < products(N); ++k) {
      constexpr unsigned I0 = 1u << 4 | (unsigned)(TM / 16) << 24;
      const Product p = product(N, k);
      mma_f16(lead, tmem + p.d0 * N,
              da + (ks * (2 * A_KO) + p.i * A_SLICE >> 4),
              db + (uint64_t)(ks * (2 * B_ROWS) + p.b * N),
              I0 | (unsigned)(p.len * N >> 3) << 17, ks || p.i || !open);
    }
}
__device__ __forceinline__ void tmem_ld4(unsigned addr, float (&v)[4]) {
  unsigned r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 4; ++i)
    v[i] = __uint_as_float(r[i]);
}

}  // namespace

// ---------------------------------------------------------------------------
// Phases.  Thread: one atom, one axis, eight consecutive n.  y and z go to
// balanced fixed-point rows [n][cos, sin][atom] (for the sums in the order
// in which a stage is read); x, times the charge, to the
// digit slices of the sums' right operand, or in FP64 to [2 n + s][atom] for
// the force's last step.
// ---------------------------------------------------------------------------
constexpr int PHN = 8;
struct PhaseArgs {
  const double *x, *y, *z, *q;
  double L[3];
  double q_unit;        // 2^62 / charge scale
  double q_lo, q_hi;    // the charges of this pass: q_lo <= |q| < q_hi
  int atom0, na, nap, kmax;
  int2 *yz;            // [2][kmax + 1][2][nap]
  unsigned char *xs;   // slices, or NULL
  double *xd;          // FP64 rows, or NULL
  int nt;              // columns per CTA
};

__global__ void __launch_bounds__(128) k_ewald_phases(PhaseArgs A) {
  const int a = blockIdx.x * 128 + threadIdx.x;  // < nap
  const int axis = blockIdx.y, n0 = blockIdx.z * PHN;
  const int nn = min(PHN, A.kmax + 1 - n0);
  const bool own = a < A.na;
  Cis e = {0, 0}, step = {0, 0};
  long long qf = 0;
  if (own) {
    const double *X = axis == 0 ? A.x : axis == 1 ? A.y : A.z;
    const unsigned long long u = turn64(X[A.atom0 + a], A.L[axis]);
    e = cis_q62(u * (unsigned long long)n0);
    step = cis_q62(u);
    if (axis == 0 && A.xs) {
      const double q = A.q[A.atom0 + a];
      qf = fabs(q) >= A.q_lo && fabs(q) < A.q_hi ? __double2ll_rn(q * A.q_unit) : 0;
    }
  }
  const int nst = A.nap / TK, piece = A.nt * 16;
  // the sums' warps read two atoms of each 8-atom group of a stage at a time:
  // those of its four groups stand side by side
  const int at = A.xs ? (a & ~31) | (a & 6) << 2 | (a >> 2 & 6) | (a & 1) : a;
  for (int i = 0; i < nn; ++i) {
    const int n = n0 + i;
    if (axis > 0) {
      int2 *row = A.yz + ((size_t)(axis - 1) * (A.kmax + 1) + n) * 2 * A.nap + at;
      row[0] = balance(e.c);
      row[A.nap] = balance(e.s);
    } else if (A.xs) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const unsigned long long w = digits_q62(mulq62(qf, s ? e.s : e.c));
        const int col = 2 * n + s, ct = col / A.nt, c = col - ct * A.nt;
        unsigned char *o = A.xs +
                           (((size_t)ct * nst + a / TK) * 4 + (a % TK) / 8) *
                               NSL * piece + c * 16 + (a % 8) * 2;
#pragma unroll
        for (int j = 0; j < NSL; ++j)
          *reinterpret_cast<__half *>(o + j * piece) =
              digit_half(w, NSL - 1 - j);
      }
    } else if (A.xd) {
      constexpr double U = 1.0 / 4611686018427387904.0;
      A.xd[(size_t)(2 * n) * A.nap + a] = (double)e.c * U;
      A.xd[(size_t)(2 * n + 1) * A.nap + a] = (double)e.s * U;
    }
    e = cis_mul(e, step);
  }
}

// ---------------------------------------------------------------------------
// The product.  FORCE false: rows = 32 pairs x 4, terms = atoms; true: rows =
// 128 atoms, terms = pairs x 4.
// ---------------------------------------------------------------------------
struct SplitArgs {
  const int2 *yz;
  int nap, kmax;
  const int *pair;  // |n_y| | |n_z| << 8 | largest n_x << 16, n_x descending
  const unsigned char *b;  // digit slices of the right operand
  int nt, nct, nst;        // columns per CTA, column tiles, stages of terms
  int per;                 // sums: stages per chunk
  int ub;                  // a CTA's outputs in units of 2^-ub
  int cut;                 // sums: bits dropped as they are added to acc
  unsigned long long *acc;  // sums: [4 pairs][nct * nt]
  // forces
  const double *xd, *q;
  const unsigned long long *cmax;  // [3][nct * nt / 2] bits of the largest
                                   // |C_w| of each n_x
  double *fpart;                   // [nct][3][n_atoms]
  int atom0, na, n_atoms;
  unsigned spin;  // polls of a wait
  int *err;
};

// binary exponent e with |c| < 2^e, for the bits of c >= 0
__device__ __forceinline__ int scale_exp(unsigned long long bits) {
  const int e = (int)(bits >> 52) - 1022;
  return bits == 0 ? 0 : max(e, -900);
}
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((long long)(e + 1023) << 52);
}
// what a column's digits are multiples of; not a number where the largest
// value is infinite or not a number
__device__ __forceinline__ double column_scale(unsigned long long bits) {
  return bits >= 0x7ff0000000000000ull ? nan("") : pow2(scale_exp(bits));
}

template <bool FORCE>
__global__ void __launch_bounds__(CTA, 1) k_ewald_split(SplitArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  // per stage buffer: operands written, products done; and the window's
  // accumulators read
  __shared__ __align__(8) uint64_t full[2], done[2], flushed;
  __shared__ unsigned tmem_base;
  __shared__ int s_bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int piece = A.nt * 16;  // bytes of one slice of 8 terms in A.b
  const int b_stage = 4 * NSL * piece, b_ring = 4 * 16 * ring_rows(A.nt);
  unsigned char *const smem_b = smem + 2 * A_STAGE;  // three stages
  const int ct = blockIdx.z;
  // columns needed where the largest n_x is nx
  auto cols = [&](int nx) {
    return min(A.nt, (max(0, 2 * (nx + 1) - ct * A.nt) + 15) & ~15);
  };
  int s0 = 0, s1 = A.nst, ntile = 0;
  if constexpr (FORCE) {
    // the first stage without a column of this tile ends the terms
    if (ct > 0) {
      int lo = 0, hi = A.nst;
      while (lo < hi) {
        const int m = (lo + hi) / 2;
        if (cols(A.pair[8 * m] >> 16) == 0)
          hi = m;
        else
          lo = m + 1;
      }
      s1 = lo;
    }
  } else {
    ntile = cols(A.pair[blockIdx.x * 32] >> 16);
    s0 = blockIdx.y * A.per;
    s1 = min(A.nst, s0 + A.per);
    if (ntile == 0 || s0 >= s1)
      return;
  }
  const int ns = s1 - s0;
  if (tid == 0) {
    s_bad = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full[i], ET / 32 + CW);
      mbar_init(&done[i], 1);
    }
    mbar_init(&flushed, ET / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == ET / 32) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
            smem_u32(&tmem_base))
        : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_base;
  // columns of the window that stage `it` (from s0) is in
  auto window_cols = [&](int it) {
    if constexpr (FORCE)
      return cols(A.pair[8 * (s0 + it / WIN * WIN)] >> 16);
    else
      return ntile;
  };
  const int grp = warp >> 2;  // columns 16 grp .. 16 grp + 15 of the outputs
  long long acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    acc[i] = 0;
  bool ok = true;
  if (warp == ET / 32) {
    // ---- the issuing warp ----
    const unsigned lead = lane == 0;
    int issued = 0;
    for (int it = 0; it < ns; ++it) {
      const int buf = it & 1;
      const bool open = it % WIN == 0;
      if (open && it)
        ok = mbar_wait(&flushed, (it / WIN - 1) & 1, &s_bad, A.spin);
      ok = ok && mbar_wait(&full[buf], (it >> 1) & 1, &s_bad, A.spin);
      if (!__all_sync(0xffffffffu, ok))
        break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned sa = smem_u32(smem + buf * A_STAGE),
                     sb = smem_u32(smem_b + it % 3 * b_ring);
      switch (window_cols(it)) {
        case 16: mma_stage<16>(lead, tmem, sa, sb, open); break;
        case 32: mma_stage<32>(lead, tmem, sa, sb, open); break;
        case 48: mma_stage<48>(lead, tmem, sa, sb, open); break;
        default: mma_stage<64>(lead, tmem, sa, sb, open); break;
      }
      if (lead)
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 "
            "[%0];" ::"r"(smem_u32(&done[buf]))
            : "memory");
      __syncwarp();
      issued = it + 1;
    }
    // nothing may be in flight when the tensor memory goes back, whatever the
    // limit of the other waits
    if (issued > 0)
      ok = mbar_wait(&done[(issued - 1) & 1], ((issued - 1) >> 1) & 1, nullptr,
                     SUMS_SPIN) &&
           ok;
    ok = ok && issued == ns;
  } else if (warp > ET / 32) {
    // ---- the right operand: stage `it` of [8-term group][slice][columns],
    // the window's columns only, into its third of a ring, each group behind
    // its slices of zeros (written anew where the window's columns differ from
    // those of the third's last stage) ----
    const int ctid = tid - ET - 32;
    const unsigned char *bsrc = A.b;
    if constexpr (FORCE)
      bsrc += (((size_t)blockIdx.y * A.nct + ct) * A.nst + s0) * b_stage;
    else
      bsrc += ((size_t)ct * A.nst + s0) * b_stage;
    auto copy = [&](int it) {
      const int n16 = window_cols(it) >> 4;
      unsigned char *const ring = smem_b + it % 3 * b_ring;
      const int z16 = zeros(16 * n16) * n16;
      if (it < 3 || n16 != window_cols(it - 3) >> 4) {
        const int nz = 16 * z16;  // 16-byte rows a group
        for (int r = ctid; r < 4 * nz; r += 32 * CW)
          reinterpret_cast<uint4 *>(ring)[r / nz * (nz + NSL * 16 * n16) + r % nz] =
              make_uint4(0, 0, 0, 0);
      }
      const unsigned dst = smem_u32(ring) + (ctid & 15) * 16;
      const unsigned char *src = bsrc + (size_t)it * b_stage + (ctid & 15) * 16;
      // 256 bytes (16 columns) at a time: piece q is group-and-slice r = q /
      // n16, block q - r n16 of the window's columns (q < 112: the division
      // by a 16-bit reciprocal is exact); the steps are independent
      const unsigned inv = 65536u / n16 + 1;
      const unsigned total = 4 * NSL * n16;
#pragma unroll
      for (int k = 0; k < (4 * NSL * NT_MAX / 16 + 2 * CW - 1) / (2 * CW); ++k) {
        const unsigned q = (ctid >> 4) + 2 * CW * k;
        const unsigned r = q * inv >> 16;
        if (q < total)
          copy16(dst + (q + (r / NSL + 1) * z16) * 256,
                 src + r * piece + (q - r * n16) * 256);
      }
    };
    if (ns > 0)
      copy(0);
    for (int it = 0; it < ns; ++it) {
      if (it >= 2)
        ok = mbar_wait(&done[it & 1], ((it - 2) >> 1) & 1, &s_bad, A.spin);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      // this stage's copies were started a stage ago
      asm volatile("cp.async.wait_all;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&full[it & 1]);
      if (it + 1 < ns)
        copy(it + 1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---- the left operand, and the accumulators ----
    // sums: four lanes take the four term groups of a row, whose factors are
    // 64 consecutive bytes: eight lanes then touch two lines (one row a lane
    // touched eight and kept the L1 tags 84 % busy); the 32 bytes beyond a
    // group's rows put the eight stores in different banks
    const int a_sub = (warp >> 2) * 8 + (lane >> 2);
    const int a_row = FORCE ? tid & 127 : (warp & 3) * 32 + a_sub;
    const int a_ko = FORCE ? tid >> 7 : lane & 3;
    const int a_off = a_ko * A_KO + (a_row >> 3) * 128 + (a_row & 7) * 16;
    const int2 *yrow = A.yz, *zrow = A.yz + (size_t)2 * (A.kmax + 1) * A.nap;
    if constexpr (FORCE) {
      yrow += blockIdx.x * TM + a_row;
      zrow += blockIdx.x * TM + a_row;
    } else {
      const int pr = A.pair[blockIdx.x * 32 + a_sub];
      const int comb = warp & 3;
      yrow += ((size_t)(pr & 255) * 2 + (comb >> 1)) * A.nap + 2 * a_ko + s0 * TK;
      zrow += ((size_t)((pr >> 8) & 255) * 2 + (comb & 1)) * A.nap + 2 * a_ko +
              s0 * TK;
    }
    // factors of the next stage, loaded while this one is formed: sums eight
    // (y, z); forces two pairs of (cos y, sin y, cos z, sin z)
    int4 ry[4], rz[4];
    int2 next = make_int2(0, 0);  // force: the pairs of the stage after
    auto load = [&](int it) {
      if constexpr (FORCE) {
        const int pp[2] = {next.x, next.y};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int2 *yp = yrow + (size_t)(pp[h] & 255) * 2 * A.nap;
          const int2 *zp = zrow + (size_t)((pp[h] >> 8) & 255) * 2 * A.nap;
          const int2 cy = __ldg(yp), sy = __ldg(yp + A.nap), cz = __ldg(zp),
                     sz = __ldg(zp + A.nap);
          ry[h] = make_int4(cy.x, cy.y, sy.x, sy.y);
          rz[h] = make_int4(cz.x, cz.y, sz.x, sz.y);
        }
        if (it + 1 < ns)
          next = __ldg(reinterpret_cast<const int2 *>(A.pair + 8 * (it + 1)) + a_ko);
      } else {
        const int4 *yp = reinterpret_cast<const int4 *>(yrow + (size_t)it * TK);
        const int4 *zp = reinterpret_cast<const int4 *>(zrow + (size_t)it * TK);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          ry[h] = __ldg(yp + 4 * h);
          rz[h] = __ldg(zp + 4 * h);
        }
      }
    };
    const unsigned trow = tmem + ((unsigned)(warp & 3) << 21) + 16 * grp;
    // add a window's accumulators to the integers (exact in FP32, see the
    // top of the file)
    auto flush = [&](int n) {
      if (16 * grp >= n)
        return;
      // multipliers of 2^-20 (times 4) and 2^-36 in units of 2^-ub, and of
      // 2^-52 (rounded half to even: a bias of every output would add up at
      // the origin, where all phases agree)
      const int drop = 52 - A.ub;
      const int m1 = 1 << (30 - drop), m2 = 1 << (16 - drop);
      const float m3 = __int_as_float((127 - drop) << 23);
      constexpr float M = 12582912.0f;  // 1.5 2^23: rounds to an integer
      constexpr int MB = 0x4B400000;    // its bits
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float v[NSL][4];
#pragma unroll
        for (int d = 0; d < NSL; ++d)
          tmem_ld4(trow + d * n + 4 * h, v[d]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // weight of v[d]: 2^(-12 - 8 d).  The low three are brought to
          // multiples of 2^-52 with a remainder of 16 bits, the integers below
          // 2^22 read from the mantissa; conversion instructions (an eighth
          // of the FP32 rate) only for v[2] and v[3].
          float c = fmaf(v[6][i], 1.0f / 256, M) - M;
          const float v5 = v[5][i] + c;
          c = fmaf(v5, 1.0f / 256, M) - M;
          const float r5 = fmaf(c, -256.0f, v5), v4 = v[4][i] + c;
          c = fmaf(v4, 1.0f / 256, M) - M;
          const float r4 = fmaf(c, -256.0f, v4);
          const int y = __float_as_int(fmaf(fmaf(r4, 256.0f, r5), m3, M)) - MB;
          const int e1 = __float2int_rn(v[2][i]) * 256 + __float2int_rn(v[3][i] + c);
          const int e0 = (__float_as_int(v[0][i] + M) - MB) * 256 +
                         (__float_as_int(v[1][i] + M) - MB);
          acc[4 * h + i] += (long long)(e0 * 4) * m1 + (long long)e1 * m2 + y;
        }
      }
    };
    if (ns > 0) {
      if constexpr (FORCE)
        next = __ldg(reinterpret_cast<const int2 *>(A.pair) + a_ko);
      load(0);
    }
    for (int it = 0; it < ns && ok; ++it) {
      unsigned char *st = smem + (it & 1) * A_STAGE;
      unsigned long long w[8];
      if constexpr (FORCE) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int2 cy = make_int2(ry[h].x, ry[h].y), sy = make_int2(ry[h].z, ry[h].w);
          const int2 cz = make_int2(rz[h].x, rz[h].y), sz = make_int2(rz[h].z, rz[h].w);
          w[4 * h + 0] = product_digits(cy, cz);
          w[4 * h + 1] = product_digits(cy, sz);
          w[4 * h + 2] = product_digits(sy, cz);
          w[4 * h + 3] = product_digits(sy, sz);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          w[2 * h] = product_digits(make_int2(ry[h].x, ry[h].y),
                                    make_int2(rz[h].x, rz[h].y));
          w[2 * h + 1] = product_digits(make_int2(ry[h].z, ry[h].w),
                                        make_int2(rz[h].z, rz[h].w));
        }
      }
      if (it + 1 < ns)
        load(it + 1);
      if (it >= 2)
        ok = mbar_wait(&done[it & 1], ((it - 2) >> 1) & 1, &s_bad, A.spin);
      if (!__all_sync(0xffffffffu, ok)) {
        ok = false;
        break;
      }
      store_slices(w, st + a_off, A_SLICE);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&full[it & 1]);
      // the last window's accumulators, when its products are done; the next
      // stage's operand is ready by then
      if (it % WIN == 0 && it) {
        ok = mbar_wait(&done[(it - 1) & 1], ((it - 1) >> 1) & 1, &s_bad, A.spin);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        flush(window_cols(it - 1));
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0)
          mbar_arrive(&flushed);
      }
    }
    if (ns > 0 && ok)
      ok = mbar_wait(&done[(ns - 1) & 1], ((ns - 1) >> 1) & 1, &s_bad, A.spin);
    if (__all_sync(0xffffffffu, ok)) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (ns > 0)
        flush(window_cols(ns - 1));
    }
  }
  if (!ok)
    *(volatile int *)&s_bad = 1;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  ok = !__syncthreads_or(!ok);
  if (warp == ET / 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(
        tmem));
  }
  if (!ok) {
    if (tid == 0)
      atomicOr(A.err, DERR_SUMS_TIMEOUT);
    return;
  }
  const int row = (warp & 3) * 32 + lane;
  if constexpr (FORCE) {
    // F_w of the row's atom: its own x phases over the columns, the four
    // column groups added in order
    double f = 0.0;
    const int a = blockIdx.x * TM + row;
    const int n0 = ct * A.nt + 16 * grp;
    const unsigned long long *cm = A.cmax + blockIdx.y * (A.nct * A.nt / 2);
    if (16 * grp < A.nt && warp < ET / 32)
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (n0 + i < 2 * (A.kmax + 1))
          f = fma((double)acc[i] * column_scale(cm[(n0 + i) / 2]),
                  A.xd[(size_t)(n0 + i) * A.nap + a], f);
    double *red = reinterpret_cast<double *>(smem);
    if (warp < ET / 32)
      red[grp * TM + row] = f;
    __syncthreads();
    if (tid < TM) {
      const int at = blockIdx.x * TM + tid;
      if (at < A.na) {
        double t = red[tid] + red[TM + tid];
        t += red[2 * TM + tid];
        t += red[3 * TM + tid];
        const double qa = A.q[A.atom0 + at];
        A.fpart[((size_t)ct * 3 + blockIdx.y) * A.n_atoms + A.atom0 + at] =
            fabs(qa) < 0.000000001 ? 0.0 : 2.0 * qa * (t * pow2(-A.ub));
      }
    }
  } else if (16 * grp < ntile && warp < ET / 32) {
    // rows are combination-major in the tile
    const int p = blockIdx.x * 32 + lane;
    unsigned long long *o = A.acc +
        ((size_t)p * 4 + (warp & 3)) * (A.nct * A.nt) + ct * A.nt + 16 * grp;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      long long v = acc[i];
      if (A.cut)  // to the nearest, halves to even
        v = (v + (1ll << (A.cut - 1)) - 1 + ((v >> A.cut) & 1)) >> A.cut;
      if (v != 0)
        atomicAdd(o + i, (unsigned long long)v);
    }
  }
}

// ---------------------------------------------------------------------------
// From D to the structure factors, in the order of the k-vectors.  Charges that
// are infinite or not a number have no digits: their terms (odd) are added here.
// ---------------------------------------------------------------------------
__global__ void k_ewald_unfold(int K, const char4 *__restrict__ kn,
                               const int *__restrict__ pair_at, int kmax,
                               const unsigned long long *__restrict__ acc,
                               int ncol, double unit, bool more, PhaseArgs odd,
                               double *sumR, double *sumI) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K)
    return;
  const char4 n = kn[k];
  const int p = pair_at[abs(n.y) * (kmax + 1) + abs(n.z)];
  const unsigned long long *d = acc + (size_t)p * 4 * ncol + 2 * n.x;
  // cos cos, cos sin, sin cos, sin sin of (y, z), with cos x and sin x; the
  // sums fit 64 bits, so wrapping partial sums do no harm
  unsigned long long c[4], s[4];
  for (int i = 0; i < 4; ++i) {
    c[i] = d[(size_t)i * ncol];
    s[i] = d[(size_t)i * ncol + 1];
  }
  const bool ny = n.y < 0, nz = n.z < 0;
  if (nz) {
    c[1] = 0 - c[1];
    s[1] = 0 - s[1];
  }
  if (ny) {
    c[2] = 0 - c[2];
    s[2] = 0 - s[2];
  }
  if (ny != nz) {
    c[3] = 0 - c[3];
    s[3] = 0 - s[3];
  }
  double re = (double)(long long)(c[0] - c[3] - s[2] - s[1]) * unit;
  double im = (double)(long long)(s[0] - s[3] + c[2] + c[1]) * unit;
  for (int a = 0; a < odd.na; ++a) {
    const double q = odd.q[a];
    if (isfinite(q))
      continue;
    const Cis e = cis_q62(turn64(odd.x[a], odd.L[0]) * (unsigned long long)n.x +
                          turn64(odd.y[a], odd.L[1]) * (unsigned long long)n.y +
                          turn64(odd.z[a], odd.L[2]) * (unsigned long long)n.z);
    re += q * (double)e.c;
    im += q * (double)e.s;
  }
  sumR[k] = more ? sumR[k] + re : re;
  sumI[k] = more ? sumI[k] + im : im;
}

// ---------------------------------------------------------------------------
// The force's right operand: C_w in FP64 with the largest value of each n_x,
// the scale of that column's digits (the digit products left out are 2^-54 of
// it per term; with one scale for all columns the forces' error was 2.7 times
// larger), then digits.
// ---------------------------------------------------------------------------
__global__ void k_pair_index(int K, const char4 *__restrict__ kn,
                             const int *__restrict__ pair_at, int kmax,
                             int npair, int *kinv) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K)
    return;
  const char4 n = kn[k];
  const int p = pair_at[abs(n.y) * (kmax + 1) + abs(n.z)];
  kinv[((size_t)n.x * npair + p) * 4 + (n.y < 0) * 2 + (n.z < 0)] = k;
}

struct CoefArgs {
  const int *kinv;
  const double *kx, *ky, *kz, *prefact, *sR, *sI;
  int npair, rows, ncol, kmax;  // rows = 4 npair
  double *coef;                 // [3][ncol][rows]
  unsigned long long *cmax;     // [3][ncol / 2], zeroed
};

__global__ void __launch_bounds__(128) k_force_coef(CoefArgs A) {
  const int p = blockIdx.x * 128 + threadIdx.x, nx = blockIdx.y;
  double c[3][8];  // [w][cos x: cc cs sc ss, sin x: cc cs sc ss]
  for (int w = 0; w < 3; ++w)
    for (int i = 0; i < 8; ++i)
      c[w][i] = 0.0;
  if (p < A.npair && nx <= A.kmax)
    for (int s = 0; s < 4; ++s) {
      const int k = A.kinv[((size_t)nx * A.npair + p) * 4 + s];
      if (k < 0)
        continue;
      const double P = A.prefact[k] * A.sR[k], Q = A.prefact[k] * A.sI[k];
      const double sy = s & 2 ? -1.0 : 1.0, sz = s & 1 ? -1.0 : 1.0;
      const double kw[3] = {A.kx[k], A.ky[k], A.kz[k]};
      for (int w = 0; w < 3; ++w) {
        const double Pw = P * kw[w], Qw = Q * kw[w];
        c[w][0] -= Qw;
        c[w][1] += sz * Pw;
        c[w][2] += sy * Pw;
        c[w][3] += sy * sz * Qw;
        c[w][4] += Pw;
        c[w][5] += sz * Qw;
        c[w][6] += sy * Qw;
        c[w][7] -= sy * sz * Pw;
      }
    }
  for (int w = 0; w < 3; ++w) {
    // the largest by its bits: infinities and NaN are above all
    unsigned long long m = 0;
    for (int i = 0; i < 8; ++i)
      m = max(m, (unsigned long long)__double_as_longlong(fabs(c[w][i])));
    for (int o = 16; o > 0; o >>= 1)
      m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0)
      atomicMax(A.cmax + w * (A.ncol / 2) + nx, m);
    if (p < A.npair)
      for (int s = 0; s < 2; ++s)
        for (int i = 0; i < 4; ++i)
          A.coef[((size_t)w * A.ncol + 2 * nx + s) * A.rows + 4 * p + i] =
              c[w][4 * s + i];
  }
}

__global__ void __launch_bounds__(128) k_force_slice(const double *__restrict__ coef,
                                                     const unsigned long long *cmax,
                                                     int rows, int ncol, int nt,
                                                     int nst, unsigned char *b) {
  const int o = blockIdx.x * 128 + threadIdx.x;  // octet of rows
  const int col = blockIdx.y, w = blockIdx.z;
  if (o >= rows / 8)
    return;
  const double *src = coef + ((size_t)w * ncol + col) * rows + 8 * o;
  const double sc = pow2(54 - scale_exp(cmax[w * (ncol / 2) + col / 2]));
  unsigned long long d[8];
  for (int i = 0; i < 8; ++i)
    d[i] = (unsigned long long)__double2ll_rn(src[i] * sc) + DIGIT_BIAS;
  const int ct = col / nt, c = col - ct * nt, piece = nt * 16;
  store_slices(d, b + ((((size_t)w * (ncol / nt) + ct) * nst + o / 4) * 4 + o % 4) *
                          NSL * piece + c * 16,
               piece);
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
namespace {

struct Shape {
  int nt, nct, ncol;
};
Shape shape_of(int kmax) {
  const int cols = 2 * (kmax + 1);
  Shape s;
  s.nct = (cols + NT_MAX - 1) / NT_MAX;
  s.nt = ((cols + s.nct - 1) / s.nct + 15) / 16 * 16;
  s.ncol = s.nt * s.nct;
  return s;
}
int stage_smem(int nt) { return 2 * A_STAGE + 3 * 4 * 16 * ring_rows(nt); }

// bits to the right of the point such that `terms` values of at most 1 fit
// 62 bits
int unit_bits(double terms) {
  return std::max(37, std::min(52, 62 - (int)std::ceil(std::log2(terms + 1.0))));
}

// bytes -> doubles of scratch, on a 128-byte boundary
size_t dbl(size_t bytes) { return (bytes + 127) / 128 * 16; }

PhaseArgs phase_args(const Box &bx, const DevBox &b, const double *x,
                     const double *y, const double *z, const Shape &sh) {
  PhaseArgs P{};
  P.x = x;
  P.y = y;
  P.z = z;
  P.q = b.q;
  for (int d = 0; d < 3; ++d)
    P.L[d] = b.L[d];
  P.kmax = b.kmax;
  P.nt = sh.nt;
  return P;
}

void launch_phases(Box &bx, PhaseArgs &P, int atom0, int na) {
  P.atom0 = atom0;
  P.na = na;
  P.nap = (na + TM - 1) / TM * TM;
  k_ewald_phases<<<dim3(P.nap / 128, 3, (P.kmax + PHN) / PHN), 128, 0,
                   bx.stream>>>(P);
}

}  // namespace

// A term is rounded to 2^-54 of its class's 2^exp (and misses digit products of
// that size), whatever its own charge, so the errors add up to 2^exp sqrt(n) for n
// charges, beside sums of sqrt(sum q^2).  A class ends where that reaches
// 8 sqrt(sum q^2) (water 1.7, where the sums' error is a sixth to a fifteenth of
// an FP64 recurrence's; with divalent ions 6.6, still one pass): smaller charges
// then have a pass of their own.  Two ions
// of 2 among 60,000 of 0.001, one pass: error 4.1e-14 of the sums' rms and 4.4e-14
// of the forces' (the FP64 kernels: 1.0e-14, 1.4e-14); two passes: 4.5e-16, 5.1e-15.
std::vector<ChargeClass> charge_classes(const std::vector<double> &q) {
  constexpr int E0 = -29;  // charges below 1e-9 are left out
  std::vector<double> n, sum;  // by exponent, from E0
  double sq = 0.0;
  for (double v : q) {
    v = std::fabs(v);
    if (!std::isfinite(v) || v < 0.000000001)
      continue;
    int e;
    std::frexp(v, &e);
    const size_t i = e - E0;
    if (i >= n.size()) {
      n.resize(i + 1, 0.0);
      sum.resize(i + 1, 0.0);
    }
    n[i] += 1.0;
    sum[i] += v;
    sq += v * v;
  }
  std::vector<ChargeClass> out;
  double count = 0.0;
  for (int i = (int)n.size() - 1; i >= 0; --i) {
    if (n[i] == 0.0)
      continue;
    const int e = i + E0;
    count += n[i];
    if (out.empty() || std::ldexp(std::sqrt(count), out.back().exp) >
                           8.0 * std::sqrt(sq)) {
      out.push_back({e, e - 1, 0.0});
      count = n[i];
    }
    out.back().bottom = e - 1;
    out.back().abs += std::ldexp(sum[i], -out.back().exp);
  }
  if (out.empty())
    out.push_back({0, 0, 0.0});
  return out;
}

// Doubles of scratch the structure factor takes.
size_t recip_sums_scratch(int n_atoms, int kmax, int npair, int batch) {
  const Shape sh = shape_of(kmax);
  const int nap = (std::min(n_atoms, batch) + TM - 1) / TM * TM;
  return dbl((size_t)4 * (kmax + 1) * nap * sizeof(int2)) +
         dbl((size_t)sh.nct * (nap / TK) * NSL * sh.nt * TK * 2) +
         dbl((size_t)npair * 4 * sh.ncol * 8);
}

int launch_recip_sums(Box &bx, const double *x, const double *y,
                      const double *z, double *sumR, double *sumI) {
  return launch_recip_sums_view(bx, bx.dev, x, y, z, sumR, sumI);
}

// The structure factor on a view: its k-vector set, its edges and the given
// coordinates.
int launch_recip_sums_view(Box &bx, const DevBox &b, const double *x,
                           const double *y, const double *z, double *sumR,
                           double *sumI) {
  const Shape sh = shape_of(b.kmax);
  const int batch = std::min(b.n_atoms, bx.cfg.sums_batch);
  const int nap = (batch + TM - 1) / TM * TM;
  const size_t b_stage = (size_t)NSL * sh.nt * TK * 2;
  const size_t d_yz = dbl((size_t)4 * (b.kmax + 1) * nap * sizeof(int2));
  const size_t d_xs = dbl((size_t)sh.nct * (nap / TK) * b_stage);
  const size_t acc_bytes = (size_t)b.npair * 4 * sh.ncol * 8;
  int rc = bx.EnsureScratch(recip_sums_scratch(b.n_atoms, b.kmax, b.npair, batch));
  if (rc)
    return rc;
  PhaseArgs P = phase_args(bx, b, x, y, z, sh);
  P.yz = (int2 *)bx.d_scratch;
  P.xs = (unsigned char *)(bx.d_scratch + d_yz);
  SplitArgs A{};
  A.yz = P.yz;
  A.kmax = b.kmax;
  A.pair = b.pair;
  A.b = P.xs;
  A.nt = sh.nt;
  A.nct = sh.nct;
  A.acc = (unsigned long long *)(bx.d_scratch + d_yz + d_xs);
  A.spin = bx.sums_spin;
  A.err = b.err;
  const size_t smem = stage_smem(sh.nt);
  raise_smem_limit((const void *)k_ewald_split<false>, smem);
  const int tiles = b.npair / 32;
  bool more = false;
  for (const ChargeClass &c : bx.q_class) {
    const int ub = unit_bits(c.abs);  // of the whole sum
    P.q_unit = std::ldexp(1.0, 62 - c.exp);
    P.q_lo = std::max(std::ldexp(1.0, c.bottom), 0.000000001);
    P.q_hi = std::ldexp(1.0, c.exp);
    if ((rc = bx.CudaCheck(cudaMemsetAsync(A.acc, 0, acc_bytes, bx.stream),
                           "memset")))
      return rc;
    for (int a0 = 0; a0 < b.n_atoms; a0 += batch) {
      launch_phases(bx, P, a0, std::min(batch, b.n_atoms - a0));
      A.nap = P.nap;
      A.nst = P.nap / TK;
      // about two CTAs per SM, of whole windows: tiles differ in their columns
      const int want = std::max(1, 2 * bx.sm_count / (tiles * sh.nct));
      A.per = ((A.nst + want - 1) / want + WIN - 1) / WIN * WIN;
      A.ub = std::max(ub, unit_bits(std::min(c.abs, (double)A.per * TK)));
      A.cut = A.ub - ub;
      k_ewald_split<false>
          <<<dim3(tiles, (A.nst + A.per - 1) / A.per, sh.nct), CTA, smem,
             bx.stream>>>(A);
    }
    P.na = bx.q_odd && !more ? b.n_atoms : 0;
    k_ewald_unfold<<<(b.K + 127) / 128, 128, 0, bx.stream>>>(
        b.K, b.kn, b.pair_at, b.kmax, A.acc, sh.ncol,
        std::ldexp(1.0, c.exp - ub), more, P, sumR, sumI);
    more = true;
  }
  return bx.CudaCheck(cudaGetLastError(), "recip sums");
}

// SetRecipRef (src/Ewald.cpp:1021-1053); sums that a wait left incomplete stay
// out of the Ref set.
__global__ void k_adopt_sums(DevBox b) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b.K || (*b.err & DERR_SUMS_TIMEOUT))
    return;
  b.sumRref[k] = b.sumRnew[k];
  b.sumIref[k] = b.sumInew[k];
}

int launch_adopt_sums(Box &bx) {
  k_adopt_sums<<<(bx.dev.K + 255) / 256, 256, 0, bx.stream>>>(bx.dev);
  return bx.CudaCheck(cudaGetLastError(), "adopt sums");
}

// Reciprocal forces without the intramolecular part into *fpart, [*nfp][3]
// [n_atoms] partials (scratch that ends `extra` doubles before its end).
int launch_force_split(Box &bx, const DevBox &b, const double *sumR,
                       const double *sumI, size_t extra, double **fpart,
                       int *nfp, double **extra_out) {
  const Shape sh = shape_of(b.kmax);
  const int batch = std::min(b.n_atoms, bx.cfg.sums_batch);
  const int nap = (batch + TM - 1) / TM * TM;
  const int rows = 4 * b.npair, nst = rows / TK;
  const size_t b_stage = (size_t)NSL * sh.nt * TK * 2;
  const size_t d_yz = dbl((size_t)4 * (b.kmax + 1) * nap * sizeof(int2));
  const size_t d_xd = dbl((size_t)sh.ncol * nap * 8);
  const size_t d_cf = dbl((size_t)3 * sh.ncol * rows * 8);
  const size_t d_sl = dbl((size_t)3 * sh.nct * nst * b_stage);
  const size_t d_fp = dbl((size_t)sh.nct * 3 * b.n_atoms * 8);
  const size_t kinv_len = (size_t)(b.kmax + 1) * b.npair * 4;
  const size_t d_ki = dbl(kinv_len * 4);
  const size_t d_cm = dbl((size_t)3 * sh.ncol / 2 * 8);
  int rc = bx.EnsureScratch(d_yz + d_xd + d_cf + d_sl + d_fp + d_ki + d_cm +
                            extra);
  if (rc)
    return rc;
  double *o = bx.d_scratch;
  PhaseArgs P = phase_args(bx, b, b.x, b.y, b.z, sh);
  P.yz = (int2 *)o;
  P.xd = o += d_yz;
  double *coef = o += d_xd;
  unsigned char *sl = (unsigned char *)(o += d_cf);
  *fpart = o += d_sl;
  int *kinv = (int *)(o += d_fp);
  unsigned long long *cmax = (unsigned long long *)(o += d_ki);
  *extra_out = o + d_cm;
  *nfp = sh.nct;
  if ((rc = bx.CudaCheck(cudaMemsetAsync(cmax, 0, d_cm * 8, bx.stream), "memset")) ||
      (rc = bx.CudaCheck(cudaMemsetAsync(kinv, 0xff, kinv_len * 4, bx.stream),
                         "memset")))
    return rc;
  k_pair_index<<<(b.K + 127) / 128, 128, 0, bx.stream>>>(
      b.K, b.kn, b.pair_at, b.kmax, b.npair, kinv);
  CoefArgs C;
  C.kinv = kinv;
  C.kx = b.kx;
  C.ky = b.ky;
  C.kz = b.kz;
  C.prefact = b.prefact;
  C.sR = sumR;
  C.sI = sumI;
  C.npair = b.npair;
  C.rows = rows;
  C.ncol = sh.ncol;
  C.kmax = b.kmax;
  C.coef = coef;
  C.cmax = cmax;
  k_force_coef<<<dim3((b.npair + 127) / 128, sh.ncol / 2), 128, 0, bx.stream>>>(C);
  k_force_slice<<<dim3((rows / 8 + 127) / 128, sh.ncol, 3), 128, 0,
                  bx.stream>>>(coef, cmax, rows, sh.ncol, sh.nt, nst, sl);
  SplitArgs A{};
  A.yz = P.yz;
  A.kmax = b.kmax;
  A.pair = b.pair;
  A.b = sl;
  A.nt = sh.nt;
  A.nct = sh.nct;
  A.nst = nst;
  A.ub = unit_bits(rows);
  A.xd = P.xd;
  A.q = b.q;
  A.cmax = cmax;
  A.fpart = *fpart;
  A.n_atoms = b.n_atoms;
  A.spin = bx.sums_spin;
  A.err = b.err;
  const size_t smem = stage_smem(sh.nt);
  raise_smem_limit((const void *)k_ewald_split<true>, smem);
  for (int a0 = 0; a0 < b.n_atoms; a0 += batch) {
    const int na = std::min(batch, b.n_atoms - a0);
    launch_phases(bx, P, a0, na);
    A.nap = P.nap;
    A.atom0 = a0;
    A.na = na;
    k_ewald_split<true><<<dim3(P.nap / TM, 3, sh.nct), CTA, smem,
                          bx.stream>>>(A);
  }
  return bx.CudaCheck(cudaGetLastError(), "reciprocal force");
}

}  // namespace gb
