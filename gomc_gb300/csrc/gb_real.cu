// Real-space kernels (FP64 plain form):
//   BoxInter        pair walk, a warp per atom, each pair once
//                   (src/CalculateEnergy.cpp:157-266); VirialCalc likewise
//   MoleculeInter   CTAs per (atom, old/new)
//                   (src/CalculateEnergy.cpp:581-686)
//   ParticleInter   CTAs per trial (src/CalculateEnergy.cpp:727-785)
//   BoxForce        pair walk from both ends, no atomics
//                   (src/CalculateEnergy.cpp:268-406)
//   MolCorrection   per molecule (src/Ewald.cpp:1056-1085)
//   CalculateTorque per molecule (src/CalculateEnergy.cpp:1365-1406)
// Partial sums land in per-CTA slots and a final single-CTA kernel adds them
// in a fixed order, so every result is reproducible run to run.
#include "gb_box.h"
#include "gb_cells.cuh"
#include "gb_pair.cuh"

namespace gb {

constexpr int RT = 128;  // threads per real-space CTA

// Sum `n` partials of width `w` (stride w) into out[0..w), fixed order.
__global__ void k_reduce_partials(const double *__restrict__ part, int n, int w,
                                  double *out) {
  __shared__ double sh[RT / 32];
  for (int c = 0; c < w; ++c) {
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += RT)
      v += part[(size_t)i * w + c];
    double r = block_sum<RT>(v, sh);
    if (threadIdx.x == 0)
      out[c] = r;
  }
}

// Column blockIdx.x of `n` partials of width w, fixed order.  The threads'
// sums are added with the rounding errors carried along (the large numbers
// meet there).
constexpr int RCT = 128;
struct Sum2 {
  double hi, lo;
};
__device__ __forceinline__ Sum2 add2(Sum2 a, double v, double lo) {
  const double s = __dadd_rn(a.hi, v), t = __dadd_rn(s, -a.hi);
  const double e = __dadd_rn(__dadd_rn(a.hi, -__dadd_rn(s, -t)),
                             __dadd_rn(v, -t));
  return {s, a.lo + (lo + e)};
}
__global__ void __launch_bounds__(RCT) k_reduce_cols(const double *__restrict__ part,
                                                     int n, int w, double *out) {
  __shared__ Sum2 sh[RCT / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Sum2 v = {0.0, 0.0};
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += RCT)
    v.hi += part[(size_t)i * w + blockIdx.x];
  for (int o = 16; o > 0; o >>= 1)
    v = add2(v, __shfl_down_sync(0xffffffffu, v.hi, o),
             __shfl_down_sync(0xffffffffu, v.lo, o));
  if (lane == 0)
    sh[warp] = v;
  __syncthreads();
  if (warp)
    return;
  v = lane < RCT / 32 ? sh[lane] : Sum2{0.0, 0.0};
  for (int o = RCT / 64; o > 0; o >>= 1)
    v = add2(v, __shfl_down_sync(0xffffffffu, v.hi, o),
             __shfl_down_sync(0xffffffffu, v.lo, o));
  if (lane == 0)
    out[blockIdx.x] = isfinite(v.lo) ? v.hi + v.lo : v.hi;
}

// ---------------------------------------------------------------------------
// The pair walk of BoxInter, VirialCalc and BoxForce.
//
// FP64 bounds all three: GB300 retires two FP64 lanes per SM and clock and a
// warp instruction costs the same with 1 active lane as with 32, so what
// counts is the number of FP64 warp instructions, and FP32 and integer work
// is 64 times cheaper.  Hence:
//   * a warp takes one atom at a time and scans the cells around it on the
//     32-bit fixed-point turns of the grid (the difference of two turns wraps
//     by itself), 32 neighbours a step, with an FP32 distance test whose
//     radius is padded beyond its rounding; survivors are compacted into a
//     queue of the warp, and FP64 runs on full batches of 32 pairs, with the
//     exact FP64 cutoff test;
//   * energies and the virial take each pair once (the 13 neighbour cells
//     after the own one in the table, which are the other 13 seen from there,
//     and later slots of the own cell: the same work for every cell), the
//     force walk takes a pair from both ends: the warp's lanes then hold one
//     atom's force, so no atomics are needed and every sum has a fixed order;
//   * comparisons of FP64 values are made on their bits, a minimum-image
//     shift is added only where a lane of the batch needs one, Lennard-Jones
//     terms are skipped for a batch without any (a hydrogen's whole walk),
//     1 / r^2 starts from the FP32 reciprocal, and of the Coulomb segment
//     polynomial degrees 0-6 are FP64 (pair_poly_at).
// One CTA of four warps takes every (grid.y * 4)-th atom of a cell; grid.y is
// set so that a warp has one atom in small boxes and up to eight in large
// ones (pair_split).  Measured on 8,000 waters, Rcut 10 A, against one CTA
// per cell pair (energies, virial) or per third of a neighbour shell
// (forces): the calls forces + reciprocal + torque 31.4 -> 24.6 ms, virial
// 15.9 -> 12.7 ms; SystemTotal of 20,000 waters 72.9 -> 70.6 ms.  Per launch
// now: forces 782 us and virial 509 us (8,000 waters), energies 776 us
// (20,000), the FP64 pipe 83 % busy (75-78 % with the last wave).
// ---------------------------------------------------------------------------
constexpr int PW = RT / 32;  // warps per CTA
constexpr int PQ = 64;       // queue slots per warp: one batch plus a scan step

// min_image on a full warp (the same result): the shift is an FP64 addition
// only for a batch in which some lane crosses half a box.
__device__ __forceinline__ double min_image_warp(double raw, double ax,
                                                 double half) {
  const bool far = (bits64(raw) & 0x7fffffffffffffffLL) > bits64(half);
  if (__any_sync(0xffffffffu, far)) {
    const double sh = far ? copysign(ax, raw) : 0.0;
    raw -= sh;
  }
  return raw;
}

// Scan constants of a box: FP32 edge of 2^-23 turns squared, and the padded
// squared cutoff.  A turn difference is cut to 23 bits (L 2^-23 at most), the
// turns themselves are within L 2^-32: the pad of 1e-6 of the longest edge
// and 1e-4 of Rcut^2 covers both.
struct Scan {
  float sx, sy, sz, cut;
};
__device__ __forceinline__ Scan scan_of(const DevBox &b, const FF &ff) {
  const float t = 1.1920929e-7f;  // 2^-23
  const float lx = (float)b.L[0] * t, ly = (float)b.L[1] * t,
              lz = (float)b.L[2] * t;
  const float rp = (float)ff.rcut + 1e-6f * fmaxf((float)b.L[0],
                                                  fmaxf((float)b.L[1],
                                                        (float)b.L[2]));
  return {lx * lx, ly * ly, lz * lz, rp * rp * 1.0001f};
}
// FP32 of a signed turn difference in units of 2^-23 turns: the top 23 bits
// placed in the mantissa of 1.5 * 2^23.
__device__ __forceinline__ float turn_f32(uint32_t a, uint32_t b) {
  return __int_as_float(0x4B400000 + ((int)(a - b) >> 9)) - 12582912.0f;
}
__device__ __forceinline__ bool scan_near(const Scan &s, const uint4 &a,
                                          const uint4 &b) {
  const float dx = turn_f32(a.x, b.x), dy = turn_f32(a.y, b.y),
              dz = turn_f32(a.z, b.z);
  return fmaf(dx * dx, s.sx, fmaf(dy * dy, s.sy, dz * dz * s.sz)) < s.cut;
}

// Whether r^2 from multiply-adds (within two units of the last place of
// dsq3's) may fall on the other side of a cutoff than dsq3's.
__device__ __forceinline__ bool beside(double distSq, double cut) {
  return (unsigned long long)(bits64(distSq) - bits64(cut) + 8) <= 16;
}

// The separation of a batch's pairs; true where the pair is inside the
// cutoff (act lanes only).  FAST: r^2 is three FP64 instructions instead of
// dsq3's five, but every cutoff is decided as by dsq3 (the walks over a box,
// which the FP64 pipe bounds: force walk of 8,000 waters 825 -> 774 us,
// energies of 20,000 862 -> 815 us; with warp_sum4 at an atom's end).
template <bool FAST>
__device__ __forceinline__ bool pair_sep(const DevBox &b, const FF &ff, bool act,
                                         const double4_32a &pi,
                                         const double4_32a &pj, double v[3],
                                         double *distSq) {
  v[0] = min_image_warp(pi.x - pj.x, b.L[0], b.half[0]);
  v[1] = min_image_warp(pi.y - pj.y, b.L[1], b.half[1]);
  v[2] = min_image_warp(pi.z - pj.z, b.L[2], b.half[2]);
  double s;
  if constexpr (FAST)
    s = fma(v[0], v[0], fma(v[1], v[1], v[2] * v[2]));
  if (!FAST || beside(s, ff.rcutSq) || beside(s, ff.rcutCoulSq))
    s = dsq3(v[0], v[1], v[2]);
  *distSq = s;
  return act && gt_pos(ff.rcutSq, s);
}

// Whether a pair's Lennard-Jones terms can be other than zero: a zero
// epsilon gives zero unless (sigma^2 / r^2)^6 overflows.
__device__ __forceinline__ bool lj_live(const FF &ff, double distSq, int idx) {
  return nonzero(ff.eps_cn[idx]) || !in_fast_range(distSq);
}

// lj_energy and lj_virial of one pair (either may be NULL), sharing 1 / r^2.
__device__ __forceinline__ void lj_terms(const FF &ff, double s, int idx,
                                         double *en, double *vir) {
  if (bits64(ff.nexp[idx]) == bits64(12.0) && in_fast_range(s)) {
    const double y = recip_cubic(s);
    // (its sixth power carries the error of sigma^2 / r^2)
    const double rRat2 = quot_pos(ff.sigmaSq[idx], s, y);
    const double attract = rRat2 * rRat2 * rRat2;
    const double repulse = attract * attract;
    if (en)
      *en = ff.eps_cn[idx] * (repulse - attract);
    if (vir)
      *vir = ff.eps_cn_6[idx] * (ff.nOver6[idx] * repulse - attract) * y;
    return;
  }
  if (en)
    *en = lj_energy(ff, s, idx);
  if (vir)
    *vir = lj_virial(ff, s, idx);
}

// Energies of one batch added to lj and re (every lane of the warp calls; re
// without QQ_FACT).
__device__ __forceinline__ void batch_energy(const DevBox &b, const FF &ff,
                                             bool act, int2 e, double &lj,
                                             double &re) {
  double4_32a pi = make_double4_32a(0, 0, 0, 0), pj = pi;
  int idx = 0;
  if (act) {
    pi = b.cell_pos[e.x];
    pj = b.cell_pos[e.y];
    idx = meta_kind(b.cell_meta[e.x]) + meta_kind(b.cell_meta[e.y]) * ff.n_kinds;
  }
  double v[3], distSq;
  const bool in = pair_sep<true>(b, ff, act, pi, pj, v, &distSq);
  if (ff.electrostatic && in) {
    const double qq = pi.w * pj.w;
    if (nonzero(qq)) {
      double p;
      if (!gt_pos(distSq, ff.rcutCoulSq) && ff.ewald &&
          pair_poly(ff, 0, distSq, &p))
        re = fma(qq, p, re);
      else
        re += coulomb_energy(ff, distSq, qq);
    }
  }
  if (in && lj_live(ff, distSq, idx)) {
    double l;
    lj_terms(ff, distSq, idx, &l, nullptr);
    lj += l;
  }
}

// Virial terms of one batch (src/CalculateEnergy.cpp:458-519): the force
// factor times the product of the atom and the molecule-centre separation;
// v6 = LJ xx, yy, zz, then Coulomb (q_i q_j, without qqFact) xx, yy, zz.
__device__ __forceinline__ void batch_virial(const DevBox &b, const FF &ff,
                                             bool act, int2 e, double v6[6]) {
  double4_32a pi = make_double4_32a(0, 0, 0, 0), pj = pi;
  int idx = 0, mi = 0, mj = 0;
  if (act) {
    pi = b.cell_pos[e.x];
    pj = b.cell_pos[e.y];
    mi = b.cell_meta[e.x];
    mj = b.cell_meta[e.y];
    idx = meta_kind(mi) + meta_kind(mj) * ff.n_kinds;
    mi = meta_mol(mi);
    mj = meta_mol(mj);
  }
  double v[3], distSq;
  const bool in = pair_sep<true>(b, ff, act, pi, pj, v, &distSq);
  double w[3];
  w[0] = v[0] * min_image_warp(b.cx[mi] - b.cx[mj], b.L[0], b.half[0]);
  w[1] = v[1] * min_image_warp(b.cy[mi] - b.cy[mj], b.L[1], b.half[1]);
  w[2] = v[2] * min_image_warp(b.cz[mi] - b.cz[mj], b.L[2], b.half[2]);
  if (ff.electrostatic && in) {
    const double qi_qj = pi.w * pj.w;
    if (nonzero(qi_qj)) {
      double p;
      if (!gt_pos(distSq, ff.rcutCoulSq) && ff.ewald &&
          pair_poly(ff, 1, distSq, &p))
        p = qi_qj * p;
      else
        p = coulomb_virial(ff, distSq, qi_qj);
      for (int d = 0; d < 3; ++d)
        v6[3 + d] = fma(p, w[d], v6[3 + d]);
    }
  }
  if (in && lj_live(ff, distSq, idx)) {
    double p;
    lj_terms(ff, distSq, idx, nullptr, &p);
    for (int d = 0; d < 3; ++d)
      v6[d] = fma(p, w[d], v6[d]);
  }
}

// Every in-range pair once: MODE 0 the energies (partials LJ, real), 1 the
// virial (six partials).
template <int MODE>
__global__ void __launch_bounds__(RT) k_box_pairs(DevBox b, const FF *__restrict__ pff,
                                                  double *part) {
  __shared__ int2 queue[PW][PQ];
  const FF &ff = *pff;
  const int c = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const Scan sc = scan_of(b, ff);
  const int n1 = b.cell_count[c];
  constexpr int NV = MODE ? 6 : 2;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k)
    v[k] = 0.0;
  int2 *q = queue[warp];
  auto eval = [&](bool act, int2 e) {
    if constexpr (MODE == 0)
      batch_energy(b, ff, act, e, v[0], v[1]);
    else
      batch_virial(b, ff, act, e, v);
  };
  int qn = 0;  // warp-uniform queue fill
  for (int s = blockIdx.y * PW + warp; s < n1; s += gridDim.y * PW) {
    const int gi = c * b.cap + s;
    const uint4 ti = b.cell_fix[gi];
    const int moli = meta_mol(b.cell_meta[gi]);
    for (int nn = NB27 / 2; nn < NB27; ++nn) {
      const int c2 = b.nbr[c * NB27 + nn];
      const int n2 = b.cell_count[c2];
      for (int j0 = nn == NB27 / 2 ? s + 1 : 0; j0 < n2; j0 += 32) {
        const int gj = c2 * b.cap + j0 + lane;
        bool in = j0 + lane < n2;
        if (in)
          in = scan_near(sc, ti, b.cell_fix[gj]) &&
               meta_mol(b.cell_meta[gj]) != moli;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in)
          q[qn + __popc(m & lt)] = make_int2(gi, gj);
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
          const int2 e = q[lane];
          const int2 mv = q[32 + lane];
          __syncwarp();
          qn -= 32;
          if (lane < qn)
            q[lane] = mv;
          __syncwarp();
          eval(true, e);
        }
      }
    }
  }
  if (qn > 0)
    eval(lane < qn, q[lane]);
  __shared__ double red[PW];
  const size_t t = (size_t)c * gridDim.y + blockIdx.y;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const double r = block_sum<RT>(v[k], red);
    if (threadIdx.x == 0)
      part[NV * t + k] = MODE == 0 && k == 1 ? r * QQ_FACT : r;
  }
}

// CTAs per cell: about 64 warps an SM in all, a warp taking one to eight
// atoms (12 to 128 warps an SM measured within 8 % of each other on 2,001 to
// 20,000 waters, 64 the best or next to it).
static int pair_split(const Box &bx, const DevBox &b) {
  const int avg = (b.n_atoms + b.ncell - 1) / b.ncell;
  const int per = std::max(1, std::min(8, b.n_atoms / (64 * bx.sm_count)));
  return std::max(1, (avg + PW * per - 1) / (PW * per));
}

template <int MODE>
static int launch_pairs(Box &bx, const DevBox &b, double *d_out,
                        const char *what) {
  constexpr int NV = MODE ? 6 : 2;
  const int split = pair_split(bx, b);
  const int n = b.ncell * split;
  int rc = bx.EnsureScratch((size_t)n * NV);
  if (rc)
    return rc;
  k_box_pairs<MODE><<<dim3(b.ncell, split), RT, 0, bx.stream>>>(b, bx.d_ff,
                                                                bx.d_scratch);
  k_reduce_cols<<<NV, RCT, 0, bx.stream>>>(bx.d_scratch, n, NV, d_out);
  return bx.CudaCheck(cudaGetLastError(), what);
}

int launch_box_virial(Box &bx, double *d_out6) {
  return launch_pairs<1>(bx, bx.dev, d_out6, "box virial");
}

int launch_box_inter(Box &bx, double *d_out2) {
  return launch_box_inter_view(bx, bx.dev, d_out2);
}

// BoxInter on a view (its coordinates, cell grid and edges).
int launch_box_inter_view(Box &bx, const DevBox &b, double *d_out2) {
  return launch_pairs<0>(bx, b, d_out2, "box inter");
}

// ---------------------------------------------------------------------------
// MoleculeInter and ParticleInter: the walk around points.  These calls are
// bound by latency -- a launch, a few dependent loads and some 25 dependent
// FP64 instructions of 64 cycles -- so there is one kernel a call: positions
// come as kernel arguments with their cells and turns (taken on the host),
// CTAs of four warps (one a sub-partition, each with its FP64 unit to itself)
// walk the 27 cells around a point with the FP32 scan and FP64 batches of the
// pair walk, and the last CTA adds the points' sums and writes them to the
// host's pinned memory.  With no more trials than SMs a trial has seven CTAs, a
// warp one cell and so one batch (2,400-sphere liquid, 10 trials: one CTA of nine
// warps a point took 14.7 us, two batches a warp and two warps a sub-partition);
// beyond, one, which fills its batches better.  us a call, seven CTAs / one: 65
// trials 34 / 39 (8,000 waters 43 / 48), 100 37 / 40 (44 / 49), 152 40 / 41
// (49 / 51), 200 45 / 42 (55 / 53), 256 51 / 42 (62 / 54).  A molecule's points
// meet in one warp of the last CTA, so there the line is 64 points: molecules of
// 33 sites 28.7 / 28.6, of 48 33.3 / 30.9, of 64 38.3 / 33.7.
// ---------------------------------------------------------------------------
constexpr int PTW = 4;       // warps per CTA
constexpr int PT_SPLIT = 7;  // CTAs per point of a call of few points
template <int N>
struct Points {
  double xyz[3 * N];
  uint32_t turn[3 * N];
  int cell[N];
};

// MOL: points 2 a and 2 a + 1 are atom a of molecule m at its own and its new
// position, the molecule itself left out, sums over all points; else point t
// is a trial position of an atom of kind ka and charge qa, sums per trial.
template <bool MOL, int N>
__global__ void __launch_bounds__(32 * PTW) k_points(DevBox b, const FF *__restrict__ pff,
                                                     const __grid_constant__ Points<N> P,
                                                     int parts, int m, int ka,
                                                     double qa, double *part,
                                                     double *out) {
  __shared__ int queue[PTW][PQ];
  __shared__ double red[2][PTW];
  const FF &ff = *pff;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int pt = blockIdx.x / parts, sub = blockIdx.x - pt * parts;
  const int i = MOL ? pt >> 1 : pt;
  const bool fresh = !MOL || (pt & 1);
  double4_32a pi = make_double4_32a(P.xyz[3 * i], P.xyz[3 * i + 1],
                                    P.xyz[3 * i + 2], qa);
  uint4 ti = make_uint4(P.turn[3 * i], P.turn[3 * i + 1], P.turn[3 * i + 2], 0);
  int cell = P.cell[i];
  if constexpr (MOL) {
    const int atom = b.mstart[m] + i;
    pi.w = b.q[atom];
    ka = b.kind[atom];
    if (!fresh) {
      pi.x = b.x[atom];
      pi.y = b.y[atom];
      pi.z = b.z[atom];
      cell = b.atom_cell[atom];
      if (cell >= 0) {
        ti = b.cell_fix[(size_t)cell * b.cap + b.atom_slot[atom]];
      } else {  // out of the grid
        cell = position_to_cell_fast(b, pi.x, pi.y, pi.z);
        ti = make_uint4(to_turns(pi.x, b.invL[0]), to_turns(pi.y, b.invL[1]),
                        to_turns(pi.z, b.invL[2]), 0);
      }
    }
  }
  const Scan sc = scan_of(b, ff);
  double lj = 0.0, re = 0.0;
  bool ovl = false;
  const double qi = pi.w * QQ_FACT;
  int *q = queue[warp];
  auto eval = [&](bool act, int gj) {
    double4_32a pj = make_double4_32a(0, 0, 0, 0);
    int idx = 0;
    if (act) {
      pj = b.cell_pos[gj];
      idx = ka + meta_kind(b.cell_meta[gj]) * ff.n_kinds;
    }
    double v[3], distSq;
    const bool in = pair_sep<false>(b, ff, act, pi, pj, v, &distSq);
    ovl |= in && fresh && gt_pos(ff.rcutLowSq, distSq);
    if (ff.electrostatic && in) {
      const double qq = qi * pj.w;
      if (nonzero(qq)) {
        double p;
        if (!gt_pos(distSq, ff.rcutCoulSq) && ff.ewald &&
            pair_poly(ff, 0, distSq, &p))
          re = fma(qq, p, re);
        else
          re += coulomb_energy(ff, distSq, qq);
      }
    }
    if (in && lj_live(ff, distSq, idx)) {
      double l;
      lj_terms(ff, distSq, idx, &l, nullptr);
      lj += l;
    }
  };
  int qn = 0;  // warp-uniform queue fill
  for (int nn = sub * PTW + warp; nn < NB27; nn += parts * PTW) {
    const int c2 = b.nbr[cell * NB27 + nn];
    const int n2 = b.cell_count[c2];
    for (int j0 = 0; j0 < n2; j0 += 32) {
      const int gj = c2 * b.cap + j0 + lane;
      bool in = j0 + lane < n2;
      if (in)
        in = scan_near(sc, ti, b.cell_fix[gj]) &&
             !(MOL && meta_mol(b.cell_meta[gj]) == m);
      const unsigned mask = __ballot_sync(0xffffffffu, in);
      if (in)
        q[qn + __popc(mask & lt)] = gj;
      qn += __popc(mask);
      __syncwarp();
      if (qn >= 32) {
        const int e = q[lane], mv = q[32 + lane];
        __syncwarp();
        qn -= 32;
        if (lane < qn)
          q[lane] = mv;
        __syncwarp();
        eval(true, e);
      }
    }
  }
  if (qn > 0)
    eval(lane < qn, q[lane]);
  const double w = warp_sum2(lj, re);
  if ((lane & 15) == 0)
    red[lane >> 4][warp] = w;
  const bool any = __syncthreads_or(ovl);
  if (warp == 0) {  // lanes 0-3 the warps' LJ, 16-19 their real space
    const int k = lane & 15;
    double v = k < PTW ? red[lane >> 4][k] : 0.0;
    for (int o = 2; o > 0; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    if (k == 0)
      part[3 * blockIdx.x + (lane >> 4)] = fresh ? v : -v;
    if (lane == 0)
      part[3 * blockIdx.x + 2] = any ? 1.0 : 0.0;
  }
  if (!last_cta((unsigned *)b.err + 2))
    return;
  const int n = gridDim.x;
  if constexpr (MOL) {
    if (warp == 0) {
      double a = 0.0, r = 0.0;
      bool o = false;
      for (int k = lane; k < n; k += 32) {
        a += __ldcg(part + 3 * k);
        r += __ldcg(part + 3 * k + 1);
        o |= __ldcg(part + 3 * k + 2) != 0.0;
      }
      const double t = warp_sum2(a, r);
      o = __any_sync(0xffffffffu, o);
      if ((lane & 15) == 0)
        out[lane >> 4] = t;
      if (lane == 0)
        out[2] = o ? 1.0 : 0.0;
    }
  } else {
    for (int k = threadIdx.x; k < 3 * (n / parts); k += 32 * PTW) {
      const double *p = part + (size_t)(k / 3) * parts * 3 + k % 3;
      double v = 0.0;
      for (int j = 0; j < parts; ++j)
        v += __ldcg(p + 3 * j);
      out[k] = v;
    }
  }
  if (threadIdx.x == 0)
    *(int *)(out + 3 * (MOL ? 1 : n / parts)) = *(volatile int *)b.err;
}

template <bool MOL, int N>
static int launch_points(Box &bx, const double *xyz, int n, int m, int kind,
                         double charge, const char *what) {
  const DevBox &b = bx.dev;
  const int pts = MOL ? 2 * n : n, parts = pts <= (MOL ? 64 : bx.sm_count) ? PT_SPLIT : 1;
  int rc = bx.EnsureScratch((size_t)3 * pts * parts);
  if (rc)
    return rc;
  Points<N> P;
  for (int i = 0; i < n; ++i) {
    for (int d = 0; d < 3; ++d) {
      P.xyz[3 * i + d] = xyz[3 * i + d];
      P.turn[3 * i + d] = to_turns(xyz[3 * i + d], b.invL[d]);
    }
    P.cell[i] = position_to_cell(b, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
  }
  k_points<MOL, N><<<pts * parts, 32 * PTW, 0, bx.stream>>>(
      b, bx.d_ff, P, parts, m, kind, charge, bx.d_scratch, bx.h_pinned);
  return bx.CudaCheck(cudaGetLastError(), what);
}

// Arguments of up to 16 positions in the small form (0.7 KB of kernel
// arguments instead of 10 KB).
int launch_mol_inter(Box &bx, int m, const double *newpos) {
  const int n = bx.host.mstart[m + 1] - bx.host.mstart[m];
  return n <= 16 ? launch_points<true, 16>(bx, newpos, n, m, 0, 0.0, "molecule inter")
                 : launch_points<true, 64>(bx, newpos, n, m, 0, 0.0, "molecule inter");
}

// ParticleInter: against every atom the cell grid holds (a molecule being
// grown by CBMC is taken out of the grid first, as in the reference).
int launch_particle_inter(Box &bx, int kind, double charge,
                          const double *trials, int ntrials) {
  return ntrials <= 16
             ? launch_points<false, 16>(bx, trials, ntrials, 0, kind, charge,
                                        "particle inter")
             : launch_points<false, 256>(bx, trials, ntrials, 0, kind, charge,
                                         "particle inter");
}

// ---------------------------------------------------------------------------
// SingleMoleculeInter: unit u = atom * 27 + neighbour cell of the atom's
// current cell; the molecule stays in the cell list and its own atoms are
// skipped (src/CalculateEnergy.cpp:1494-1556).  lam = old VDW, new VDW, old
// Coulomb, new Coulomb; partials = old LJ, old real, new LJ, new real.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RT) k_single_mol_inter(
    DevBox b, const FF *__restrict__ pff, int m,
    const double *__restrict__ lam, double *part) {
  const FF &ff = *pff;
  int u = blockIdx.x;
  int a = u / NB27, n = u % NB27;
  int atom = b.mstart[m] + a;
  double px = b.x[atom], py = b.y[atom], pz = b.z[atom];
  int cell = position_to_cell_fast(b, px, py, pz);
  int c2 = b.nbr[cell * NB27 + n];
  int n2 = b.cell_count[c2];
  double qa = b.q[atom];
  int ka = b.kind[atom];
  double lov = lam[0], lnv = lam[1], loc = lam[2], lnc = lam[3];
  double ljo = 0.0, reo = 0.0, ljn = 0.0, ren = 0.0;
  for (int j = threadIdx.x; j < n2; j += RT) {
    size_t s = (size_t)c2 * b.cap + j;
    int mj = b.cell_meta[s];
    if (meta_mol(mj) == m)
      continue;
    double4_32a pj = b.cell_pos[s];
    double dx = min_image(px - pj.x, b.L[0], b.half[0]);
    double dy = min_image(py - pj.y, b.L[1], b.half[1]);
    double dz = min_image(pz - pj.z, b.L[2], b.half[2]);
    double distSq = dsq3(dx, dy, dz);
    if (!(ff.rcutSq > distSq))
      continue;
    int idx = ka + meta_kind(mj) * ff.n_kinds;
    if (ff.electrostatic) {
      double qq = qa * pj.w * QQ_FACT;
      if (qq != 0.0) {
        ren += coulomb_energy_lambda(ff, distSq, idx, qq, lnc);
        reo += coulomb_energy_lambda(ff, distSq, idx, qq, loc);
      }
    }
    ljn += lj_energy_lambda(ff, distSq, idx, lnv);
    ljo += lj_energy_lambda(ff, distSq, idx, lov);
  }
  __shared__ double red[RT / 32];
  double v[4] = {ljo, reo, ljn, ren};
  for (int c = 0; c < 4; ++c) {
    double r = block_sum<RT>(v[c], red);
    if (threadIdx.x == 0)
      part[4 * u + c] = r;
  }
}

int launch_single_mol_inter(Box &bx, int m, const double *d_lam4,
                            double *d_out4) {
  int na = bx.host.mstart[m + 1] - bx.host.mstart[m];
  int units = na * NB27;
  int rc = bx.EnsureScratch((size_t)units * 4);
  if (rc)
    return rc;
  k_single_mol_inter<<<units, RT, 0, bx.stream>>>(bx.dev, bx.d_ff, m, d_lam4,
                                                  bx.d_scratch);
  k_reduce_partials<<<1, RT, 0, bx.stream>>>(bx.d_scratch, units, 4, d_out4);
  return bx.CudaCheck(cudaGetLastError(), "single molecule inter");
}

// ---------------------------------------------------------------------------
// Ewald intramolecular correction, one thread per molecule
// ---------------------------------------------------------------------------
__global__ void k_correction(DevBox b, const FF *__restrict__ pff, double *part) {
  const FF &ff = *pff;
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  double corr = 0.0;
  if (m < b.n_mol) {
    int a0 = b.mstart[m], n = b.mstart[m + 1] - a0;
    for (int i = 0; i < n; i++) {
      if (fabs(b.q[a0 + i]) < 0.000000001)
        continue;
      for (int j = i + 1; j < n; j++) {
        int p = a0 + i, q = a0 + j;
        double dx = min_image(b.x[p] - b.x[q], b.L[0], b.half[0]);
        double dy = min_image(b.y[p] - b.y[q], b.L[1], b.half[1]);
        double dz = min_image(b.z[p] - b.z[q], b.L[2], b.half[2]);
        double distSq = dsq3(dx, dy, dz);
        double dist = sqrt(distSq);
        corr += (b.q[p] * b.q[q] * erf(ff.alpha * dist) / dist);
      }
    }
    corr = -1.0 * QQ_FACT * corr;
  }
  __shared__ double red[RT / 32];
  double s = block_sum<RT>(corr, red);
  if (threadIdx.x == 0)
    part[blockIdx.x] = s;
}

int launch_correction(Box &bx, double *d_out) {
  int nb = (bx.dev.n_mol + RT - 1) / RT;
  int rc = bx.EnsureScratch(nb);
  if (rc)
    return rc;
  k_correction<<<nb, RT, 0, bx.stream>>>(bx.dev, bx.d_ff, bx.d_scratch);
  k_reduce_partials<<<1, RT, 0, bx.stream>>>(bx.d_scratch, nb, 1, d_out);
  return bx.CudaCheck(cudaGetLastError(), "correction");
}

// ---------------------------------------------------------------------------
// BoxForce: the pair walk from both ends.  A warp's lanes hold partial forces
// on its atom, added over the warp in a fixed order; energies count the pairs
// that k_box_pairs takes.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(RT) k_box_force(DevBox b, const FF *__restrict__ pff,
                                                  double *aF, double *epart) {
  __shared__ unsigned queue[PW][PQ];
  const FF &ff = *pff;
  const int c = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const Scan sc = scan_of(b, ff);
  const int n1 = b.cell_count[c];
  double lj = 0.0, re = 0.0;
  unsigned *q = queue[warp];
  for (int s = blockIdx.y * PW + warp; s < n1; s += gridDim.y * PW) {
    const int gi = c * b.cap + s;
    const uint4 ti = b.cell_fix[gi];
    const double4_32a pi = b.cell_pos[gi];
    const int mi = b.cell_meta[gi];
    const int moli = meta_mol(mi), ki = meta_kind(mi);
    const double qi = pi.w * QQ_FACT;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    // one batch: entries are slot << 1 | (the pair's energy is counted here)
    auto eval = [&](bool act, unsigned e) {
      const int gj = (int)(e >> 1);
      const bool first = act && (e & 1);
      double4_32a pj = make_double4_32a(0, 0, 0, 0);
      int idx = 0;
      if (act) {
        pj = b.cell_pos[gj];
        idx = ki + meta_kind(b.cell_meta[gj]) * ff.n_kinds;
      }
      double v[3], distSq;
      const bool in = pair_sep<true>(b, ff, act, pi, pj, v, &distSq);
      double f = 0.0;
      const bool table = in && !gt_pos(distSq, ff.rcutCoulSq) && ff.ewald;
      if (ff.electrostatic && in) {
        const double qq = qi * pj.w;
        if (nonzero(qq)) {
          double p, e = 0.0;
          if (table && pair_poly(ff, 1, distSq, &p)) {
            f = qq * p;
            if (first && pair_poly(ff, 0, distSq, &e))
              re = fma(qq, e, re);
          } else {
            f = coulomb_virial(ff, distSq, qq);
            if (first)
              re += coulomb_energy(ff, distSq, qq);
          }
        }
      }
      if (in && lj_live(ff, distSq, idx)) {
        double l, p;
        lj_terms(ff, distSq, idx, &l, &p);
        if (first)
          lj += l;
        f += p;
      }
      if (in) {
        fx = fma(v[0], f, fx);
        fy = fma(v[1], f, fy);
        fz = fma(v[2], f, fz);
      }
    };
    int qn = 0;  // warp-uniform queue fill
    for (int nn = 0; nn < NB27; ++nn) {
      const int c2 = b.nbr[c * NB27 + nn];
      const int n2 = b.cell_count[c2];
      for (int j0 = 0; j0 < n2; j0 += 32) {
        const int j = j0 + lane, gj = c2 * b.cap + j;
        bool in = j < n2;
        if (in)
          in = scan_near(sc, ti, b.cell_fix[gj]) &&
               meta_mol(b.cell_meta[gj]) != moli;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in)
          q[qn + __popc(m & lt)] =
              (unsigned)gj << 1 | (nn > NB27 / 2 || (nn == NB27 / 2 && j > s) ? 1u : 0u);
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
          const unsigned e = q[lane], mv = q[32 + lane];
          __syncwarp();
          qn -= 32;
          if (lane < qn)
            q[lane] = mv;
          __syncwarp();
          eval(true, e);
        }
      }
    }
    if (qn > 0)
      eval(lane < qn, q[lane]);
    __syncwarp();  // the queue is read before the next atom fills it
    const double v4[4] = {fx, fy, fz, 0.0};
    const double f = warp_sum4(v4);
    if ((lane & 7) == 0 && lane < 24)
      aF[3 * (size_t)b.cell_atom[gi] + (lane >> 3)] = f;
  }
  __shared__ double red[PW];
  const double A = block_sum<RT>(lj, red);
  const double R = block_sum<RT>(re, red);
  if (threadIdx.x == 0) {
    const size_t t = (size_t)c * gridDim.y + blockIdx.y;
    epart[2 * t] = A;
    epart[2 * t + 1] = R;
  }
}

__global__ void k_mol_force(DevBox b, const double *__restrict__ aF, double *mF) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= b.n_mol)
    return;
  double f[3] = {0, 0, 0};
  for (int a = b.mstart[m]; a < b.mstart[m + 1]; ++a)
    for (int d = 0; d < 3; ++d)
      f[d] += aF[3 * (size_t)a + d];
  for (int d = 0; d < 3; ++d)
    mF[3 * (size_t)m + d] = f[d];
}

int launch_mol_force(Box &bx, const DevBox &b, const double *aF, double *mF) {
  k_mol_force<<<(b.n_mol + 127) / 128, 128, 0, bx.stream>>>(b, aF, mF);
  return bx.CudaCheck(cudaGetLastError(), "molecule forces");
}

int launch_box_force(Box &bx, const DevBox &b, double *aF, double *mF,
                     double *d_out2) {
  const int split = pair_split(bx, b);
  const int n = b.ncell * split;
  int rc = bx.EnsureScratch((size_t)n * 2);
  if (rc)
    return rc;
  k_box_force<<<dim3(b.ncell, split), RT, 0, bx.stream>>>(b, bx.d_ff, aF,
                                                          bx.d_scratch);
  if ((rc = launch_mol_force(bx, b, aF, mF)))
    return rc;
  k_reduce_cols<<<2, RCT, 0, bx.stream>>>(bx.d_scratch, n, 2, d_out2);
  return bx.CudaCheck(cudaGetLastError(), "box force");
}

// ---------------------------------------------------------------------------
// CalculateTorque: molecule torque from atom forces (real + reciprocal)
// ---------------------------------------------------------------------------
__global__ void k_torque(DevBox b, const double *__restrict__ aF,
                         const double *__restrict__ aR, double *tq) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= b.n_mol)
    return;
  double tx = 0, ty = 0, tz = 0;
  for (int p = b.mstart[m]; p < b.mstart[m + 1]; ++p) {
    double d0 = min_image(b.x[p] - b.cx[m], b.L[0], b.half[0]);
    double d1 = min_image(b.y[p] - b.cy[m], b.L[1], b.half[1]);
    double d2 = min_image(b.z[p] - b.cz[m], b.L[2], b.half[2]);
    double f0 = aF[3 * (size_t)p] + aR[3 * (size_t)p];
    double f1 = aF[3 * (size_t)p + 1] + aR[3 * (size_t)p + 1];
    double f2 = aF[3 * (size_t)p + 2] + aR[3 * (size_t)p + 2];
    tx += d1 * f2 - d2 * f1;
    ty += d2 * f0 - d0 * f2;
    tz += d0 * f1 - d1 * f0;
  }
  tq[3 * (size_t)m] = tx;
  tq[3 * (size_t)m + 1] = ty;
  tq[3 * (size_t)m + 2] = tz;
}

int launch_torque(Box &bx, const DevBox &d, const double *aF,
                  const double *aR, double *tq) {
  k_torque<<<(d.n_mol + 127) / 128, 128, 0, bx.stream>>>(d, aF, aR, tq);
  return bx.CudaCheck(cudaGetLastError(), "torque");
}

}  // namespace gb
