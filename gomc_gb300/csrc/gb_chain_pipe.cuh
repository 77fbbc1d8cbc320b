// FP64 move chain with two moves in flight (included by gb_mc.cu, after
// k_chain_fp64, whose helpers and layout it shares).
//
// The chain of k_chain_fp64 spends about half of a move waiting: the last
// partial reaches the deciding CTA, the sums, the decision, its release
// store and its way back to every CTA take about as long as the CTAs' own
// phase A.  Here one CTA (the last) does nothing but decide, and the other
// G - 1 CTAs ("work CTAs") start move t + 1 as soon as their partials of
// move t are out, while move t is being decided.  Move t + 1's energy
// depends on move t's outcome in two places only, and a work CTA evaluates
// both outcomes:
//   * reciprocal space: the new sums of move t + 1 on the committed
//     structure factors (t rejected) and on move t's new sums (t
//     accepted), both kept, one of them chosen at the commit -- the same
//     additions, in the same order, as the chain that waits;
//   * real space: the atoms of move t's molecule that the CTA owns, at
//     their old and at their new positions, against move t + 1's molecule
//     (all other own atoms are the same on both outcomes).
// Each work CTA stores two sets of partials (one per outcome of the
// previous move); the decider reads the set its own previous decision
// names.  Move t + 1 does not run ahead of move t's decision when it moves
// the same molecule as move t or as move t - 1 while that one is still
// undecided, or follows a settings adjustment: then move t's decision is
// waited for, committed, and move t + 1's context is built behind a grid
// barrier (as in k_chain_fp64).
//
// Ordering (acquire/release on the decision word and the context flags):
//   * work CTA at move t: phase A(t) -> partials(t) -> decision(t - 1)
//     and the flags of context(t + 1), in one poll -> commit(t - 1) ->
//     phase A(t + 1);
//   * decider at move t: CTA 0's flag of context(t) -> header -> every
//     work CTA's partials(t) -> decision -> the word -> partial slots reset,
//     coordinates written -> fence (it releases them with the next word).
// Contexts rotate over four buffers and partials over three slot sets: a
// writer overwrites context t - 2's buffer while building context t + 2 in
// phase A(t), after it has seen decision t - 2, which the decider gave only
// after every work CTA had read context t - 2 and stored partials(t - 2) (and
// had read that context's header itself); a work CTA stores
// partials(t + 3) after it has seen decision t + 1, behind which the
// decider reset slot set t.  The decider can run at most one move past a
// work CTA's read of the word.
// No counterpart in the reference (its moves are sequential,
// src/moves/Translate.h:97-138, src/moves/Rotation.h:89-130).

// The decision word of move t: ((t + 1) << 4) | the outcomes of moves t,
// t - 1, t - 2, t - 3 in bits 0..3, so that one load of it gives a work
// CTA the outcome of a move the decider has already passed.
__device__ __forceinline__ unsigned dec_word(int t, unsigned hist) {
  return ((unsigned)(t + 1) << 4) | (hist & 15u);
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(unsigned *p, unsigned v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// integers in the order of finite FP64 values
__device__ __forceinline__ long long order64(double v) {
  const long long i = __double_as_longlong(v);
  return i ^ ((i >> 63) & 0x7fffffffffffffffLL);
}
// the outcome of move tt from a word at or past it (at most three moves)
__device__ __forceinline__ int dec_outcome(unsigned w, int tt) {
  return (int)((w >> ((int)(w >> 4) - (tt + 1))) & 1u);
}

// Dynamic shared memory of one CTA of k_chain_fp64_pipe (the layout of
// k_chain_fp64 with four k-chunk buffers and the atoms spread over the
// work CTAs).
__host__ __device__ inline size_t chain_pipe_kvec_doubles(int kc_max) {
  return ((9 * (size_t)kc_max + (kc_max + 1) / 2 + 1) & ~(size_t)1);
}

// The pair list of a k-chunk CTA: one segment of PSEG entries per listing
// warp and one for the previous move's atoms, so that the list needs one CTA
// barrier and no CTA-wide prefix sum.
constexpr int PSEG = 64;
constexpr int PNSEG = CT / 32;
constexpr int ICL_CAP = PSEG * PNSEG;

// Minimum-image wrap of one axis decided on fixed-point turns when a pair
// is listed: 1 for -L, 2 for +L (2 bits per axis).  Only a pair near half a
// box edge apart -- far outside the cutoff -- could be decided otherwise
// than by the FP64 test of BoxDimensions::MinImage.
__device__ __forceinline__ unsigned turn_wrap(const uint32_t *tp, uint4 f) {
  const uint32_t tf[3] = {f.x, f.y, f.z};
  unsigned w = 0;
  for (int d = 0; d < 3; ++d) {
    const unsigned dt = tp[d] - tf[d];
    if (tp[d] > tf[d] ? dt > 0x80000000u : -dt > 0x80000000u)
      w |= (tp[d] > tf[d] ? 1u : 2u) << (2 * d);
  }
  return w;
}

// The force field's pair tables held in shared memory by the chain with two
// moves in flight: the erfc(alpha r)/r segments in the layout of FF::pair_tab
// without the force factors (NULL: read from global memory) and the LJ
// sigma^2 and epsilon C_n of every kind pair.
struct PairTabs {
  const double *etab;
  const double *sig2, *eps;
};

// Terms outside the fast forms (exponents other than 12, r^2 outside the
// tables), called rather than inlined: the chain's phases stay short enough
// for the instruction cache.
__device__ __noinline__ double lj_energy_far(const FF *ff, double s, int idx) {
  return lj_energy(*ff, s, idx);
}
__device__ __noinline__ double erfc_over_r_far(const FF *ff, double s) {
  return erfc_over_r(*ff, s);
}

// erfc(alpha r) / r from the segments in shared memory
__device__ __forceinline__ double erfc_over_r_tab(const FF &ff,
                                                  const double *tab, double s) {
  const long long bits = bits64(s);
  const int seg = (int)(bits >> 46) - ff.etab_key0;
  if (tab == nullptr || (unsigned)seg >= (unsigned)ff.etab_nseg)
    return erfc_over_r_far(&ff, s);
  const double2 *c = (const double2 *)(tab + (size_t)seg * 8);
  return pair_poly_at(bits, c[0], c[1], c[2], c[3]);
}

// One pair's terms, with fewer FP64 instructions than pair_term (a warp's FP64
// instruction holds its SM sub-partition's FP64 unit for about 64 cycles on
// GB300, so their count sets the time of a pass over the pair list): the minimum
// image from the listed wrap bits (the same FP64 differences: x - L is x + (-L)),
// added only where a lane has one; the neighbour's charge stored times QQ_FACT;
// comparisons on the bits; degrees 7 and 8 of the erfc(alpha r)/r segment in FP32
// (pair_poly_at); and -- where every kind pair has the 12-6 form -- sigma^2 / r^2
// as a product with recip_cubic, for pairs with an epsilon.
// Signed for the side (new position +, old -): false outside the cutoff.  a, side: the moved atom and whether its new position;
// pzq: the neighbour's z and charge times QQ_FACT.
__device__ __forceinline__ bool pair_energy_pipe(const ChainArgs &A,
                                                 const double *hdr, int a,
                                                 int side, double2 pxy,
                                                 double2 pzq, int mj,
                                                 unsigned wrap,
                                                 bool lj12, bool coul_cut,
                                                 const PairTabs &pt, double &e,
                                                 double &l, bool &ov) {
  const DevBox &b = A.b;
  const FF &ff = *A.ff;
  const double *pp = hdr + (side ? 48 : 24) + 3 * a;
  double dx = pp[0] - pxy.x, dy = pp[1] - pxy.y, dz = pp[2] - pzq.x;
  if (wrap & 3u)
    dx += (wrap & 1u) ? -b.L[0] : b.L[0];
  if (wrap & 12u)
    dy += (wrap & 4u) ? -b.L[1] : b.L[1];
  if (wrap & 48u)
    dz += (wrap & 16u) ? -b.L[2] : b.L[2];
  const double d2 = dsq3(dx, dy, dz);
  if (!gt_pos(ff.rcutSq, d2))
    return false;
  ov = side && gt_pos(ff.rcutLowSq, d2);
  e = 0.0;
  if (ff.electrostatic && !(coul_cut && gt_pos(d2, ff.rcutCoulSq))) {
    const double qq = hdr[108 + a] * pzq.y;
    e = ff.ewald ? qq * erfc_over_r_tab(ff, pt.etab, d2) : qq / sqrt(d2);
  }
  const int idx = ((const int *)(hdr + 116))[a] + meta_kind(mj) * ff.n_kinds;
  if (lj12 && in_fast_range(d2)) {
    l = 0.0;
    const double eps = pt.eps[idx];
    if (bits64(eps) != 0) {
      const double rRat2 = pt.sig2[idx] * recip_cubic(d2);
      const double attract = rRat2 * rRat2 * rRat2;
      l = eps * fma(attract, attract, -attract);
    }
  } else {
    l = lj_energy_far(&ff, d2, idx);
  }
  // the old position's terms subtracted: the sign bit flipped (exact)
  const unsigned long long neg = side ? 0ull : 0x8000000000000000ull;
  e = __longlong_as_double((long long)((unsigned long long)__double_as_longlong(e) ^ neg));
  l = __longlong_as_double((long long)((unsigned long long)__double_as_longlong(l) ^ neg));
  return true;
}

// pair_energy_pipe added to one set of sums (a pair past a full list)
__device__ __noinline__ void pair_term_pipe(const ChainArgs &A,
                                            const double *hdr, int a,
                                            int side, double2 pxy,
                                            double2 pzq, int mj,
                                            unsigned wrap, bool lj12,
                                            bool coul_cut, const PairTabs &pt,
                                            double &lj, double &re,
                                            double &ovl) {
  double e, l;
  bool ov;
  if (pair_energy_pipe(A, hdr, a, side, pxy, pzq, mj, wrap, lj12, coul_cut, pt,
                       e, l, ov)) {
    re += e;
    lj += l;
    if (ov)
      ovl = 1.0;
  }
}

__global__ void __launch_bounds__(CT, 1) k_chain_fp64_pipe(ChainArgs A) {
  extern __shared__ double dyn[];
  __shared__ ChainShared S;
  __shared__ double red6[6][CT / 32];     // warp sums, both outcomes
  const DevBox &b = A.b;
  const FF &ff = *A.ff;
  const int G = gridDim.x, cta = blockIdx.x;
  const int W = G - 1;  // work CTAs 0 .. W - 1; CTA W decides
  const bool leader = cta == W;
  const int nkb = A.nkless;
  const int kG = W - nkb;
  const int kc_max = (b.K + kG - 1) / kG;
  const bool kless = cta < nkb;
  const int kbeg = (kless || leader) ? b.K : min(b.K, (cta - nkb) * kc_max);
  const int kc = (kless || leader) ? 0 : min(kc_max, b.K - kbeg);
  const int pw = kless ? 0 : 3;  // the warp that evaluates the pair terms
  // k-chunk buffers [4][re, im][kc_max]: the committed structure factors,
  // the previous move's new sums while it is undecided, and this move's new
  // sums on either outcome of the previous one (the roles rotate)
  double *const kbuf = dyn;
  auto KR = [&](int i) { return kbuf + (size_t)(2 * i) * kc_max; };
  auto KI = [&](int i) { return kbuf + (size_t)(2 * i + 1) * kc_max; };
  double *const pf = dyn + 8 * (size_t)kc_max;
  char4 *const kn = (char4 *)(pf + kc_max);
  const int stride = b.kmax + 1;
  // phase rows of this move and, prefetched, of the next (the roles swap)
  double2 *const tab0 = (double2 *)(dyn + chain_pipe_kvec_doubles(kc_max));
  double2 *const tab1 = tab0 + (size_t)(2 * MAX_MOL_ATOMS * 3) * stride;
  double2 *tab = tab0;
  double2 *const exy = tab1 + (size_t)(2 * MAX_MOL_ATOMS * 3) * stride;
  unsigned short *const pidx =
      (unsigned short *)(exy + NPAIR_CAP * 2 * MAX_MOL_ATOMS);
  // The atoms are owned by the work CTAs with a k-chunk (the context
  // writers without one build the next context instead), through a
  // multiplicative permutation of the atom index (p = a * perm_m mod
  // n_atoms): atom a by CTA nkb + p % OWN, at index p / OWN of its share.
  // Atom indices follow the build order of the system (a lattice, at
  // first), so without the permutation the atoms near a molecule can crowd
  // onto a few CTAs and lengthen their pair lists.
  const int OWN = W - nkb;
  // x mod n_atoms by Barrett reduction (perm_r = floor((2^64 - 1) / n)):
  // integer multiplies only, no 64-bit division
  auto mod_n = [&](unsigned long long x) {
    const unsigned long long n = (unsigned long long)b.n_atoms;
    unsigned long long r = x - __umul64hi(x, A.perm_r) * n;
    return (int)(r >= n ? r - n : r);
  };
  const int orank = cta - nkb;  // this CTA's rank among the owners
  const int own_per = (b.n_atoms + OWN - 1) / OWN;
  const int on = (!leader && orank >= 0 && orank < b.n_atoms)
                     ? (b.n_atoms - orank + OWN - 1) / OWN
                     : 0;
  double2 *const oxy =
      (double2 *)(((uintptr_t)(pidx + kc_max) + 15) & ~(uintptr_t)15);
  double2 *const ozq = oxy + own_per;
  uint4 *const ot = (uint4 *)(ozq + own_per);
  // the erfc(alpha r)/r segments after them (k-chunk CTAs, Ewald on)
  double *const etab_s = (double *)(ot + own_per);
  __shared__ double lj_sig2_s[MAX_KINDS * MAX_KINDS];
  __shared__ double lj_eps_s[MAX_KINDS * MAX_KINDS];
  __shared__ char2 pair_n[NPAIR_CAP];
  __shared__ int npair;
  int bS = 0, bP = -1;  // committed and pending k-chunk buffers
  for (int i = threadIdx.x; i < kc; i += CT) {
    int k = kbeg + i;
    KR(0)[i] = b.sumRref[k];
    KI(0)[i] = b.sumIref[k];
    pf[i] = b.prefact[k];
    kn[i] = b.kn[k];
  }
  for (int i = threadIdx.x; i < on; i += CT) {
    const int a = mod_n((unsigned long long)(orank + OWN * i) * A.perm_minv);
    const double x = b.x[a], y = b.y[a], z = b.z[a];
    oxy[i] = make_double2(x, y);
    ozq[i] = make_double2(z, b.q[a] * QQ_FACT);  // the charge times QQ_FACT
    ot[i] = make_uint4(to_turns(x, b.invL[0]), to_turns(y, b.invL[1]),
                       to_turns(z, b.invL[2]),
                       (unsigned)pack_meta(b.mol[a], b.kind[a]));
  }
  const bool own_tab = !leader && !kless && ff.pair_tab != nullptr;
  if (own_tab)
    for (int i = threadIdx.x; i < ff.etab_nseg * 8; i += CT)
      etab_s[i] = ff.pair_tab[(i >> 3) * 16 + (i & 7)];
  for (int i = threadIdx.x; i < ff.n_kinds * ff.n_kinds; i += CT) {
    lj_sig2_s[i] = ff.sigmaSq[i];
    lj_eps_s[i] = ff.eps_cn[i];
  }
  const PairTabs ptab{own_tab ? etab_s : nullptr, lj_sig2_s, lj_eps_s};
  __shared__ int lj12_sh;
  if (threadIdx.x == 0) {
    int all12 = 1;
    for (int i = 0; i < ff.n_kinds * ff.n_kinds; ++i)
      all12 &= ff.eps_cn[i] == 0.0 || ff.nexp[i] == 12.0;
    lj12_sh = all12;
    S.last_m = -1;
    S.last_acc = 0;
    S.set = *A.set;
    for (int i = 0; i < 5; ++i)
      S.e_run[i] = b.energy[i];
    S.gen = ld_acquire(&A.bar[1]);
  }
  __syncthreads();
  if (threadIdx.x == 0)
    npair = chunk_columns(kn, kc, pair_n, pidx);
  __syncthreads();

  const int total_threads = G * CT;
  const int gtid = cta * CT + threadIdx.x;
  const bool lj12 = lj12_sh != 0;
  const bool coul_cut = ff.rcutCoulSq < ff.rcutSq;
  const float turn_f[3] = {(float)(b.L[0] * 2.3283064365386963e-10),
                           (float)(b.L[1] * 2.3283064365386963e-10),
                           (float)(b.L[2] * 2.3283064365386963e-10)};
  const float cut_f = (float)(ff.rcutSq * 1.0001);
  auto make_props = [&](int t0) {
    int t1 = t0;
    while (t1 < A.n) {
      long long step = A.first + t1;
      if (t1 > t0 && (step + 1) % S.set.adj == 0)
        break;
      ++t1;
    }
    for (int t = t0 + gtid; t < t1; t += total_threads)
      make_proposal(A.moves[t], S.set, A.prop + (size_t)t * 12);
  };

  // prologue: the first block's proposals and context 0
  if (threadIdx.x == 0)
    settings_adjust(S.set, A.first);
  __syncthreads();
  make_props(0);
  if (!grid_sync(A.bar, G, S.gen, b.err, &S.flag, A.spin))
    return;
  build_ctx(A, S, 0, nullptr, 0, 0, CT);
  if (!grid_sync(A.bar, G, S.gen, b.err, &S.flag, A.spin))
    return;

  // the profiled work CTA: the first with a k-chunk (the context writers
  // before it only build contexts)
  const int pslot = cta == nkb ? 0 : leader ? 1 : -1;
  const bool prof = A.prof && threadIdx.x == 0 && pslot >= 0;
  long long pacc[5] = {0, 0, 0, 0, 0};
  long long tclk = prof ? clock64() : 0;
  auto mark = [&](int ph) {
    if (prof) {
      long long now = clock64();
      pacc[ph] += now - tclk;
      tclk = now;
    }
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the settings adjustment before a move (the next move's proposals are
  // made after it), behind a grid barrier; false when a wait gave up
  auto adjust_before = [&](int t1, bool bnd) -> bool {
    long long step = A.first + t1;
    if (!bnd)
      return true;
    __syncthreads();
    if (threadIdx.x == 0)
      settings_adjust(S.set, step);
    __syncthreads();
    make_props(t1);
    return grid_sync(A.bar, G, S.gen, b.err, &S.flag, A.spin);
  };
  int nmol = A.n > 1 ? A.moves[1].mol : -1;
  // (first + t + 2) mod AdjSteps, carried from move to move (no 64-bit
  // division per move): zero where a settings adjustment precedes move
  // t + 1
  int adj_r = (int)((A.first + 2) % S.set.adj);

  if (leader) {
    // ---------------- the deciding CTA ----------------
    bool pend = false;
    int m_prev = -1, acc_prev = 0;
    unsigned hist = 0;  // outcomes of the last moves, newest in bit 0
    const double nbeta = -ff.beta;
    for (int t = 0; t < A.n; ++t) {
      const int mol_next = nmol;
      nmol = t + 2 < A.n ? A.moves[t + 2].mol : -1;
      const bool bnd = adj_r == 0;
      adj_r = adj_r + 1 == S.set.adj ? 0 : adj_r + 1;
      // this move's header: complete once CTA 0 has flagged the context
      // when it was built during the previous move's phase A, and behind
      // the last grid barrier otherwise
      if (threadIdx.x == 0)
        S.ok = pend ? wait_geq(A.seq + SEQ_CTX, (unsigned)t, b.err, A.spin)
                    : 1;
      __syncthreads();
      if (!S.ok)
        return;
      const double *ctx_t = A.ctx + (size_t)(t % PIPE_NCTX) * A.ctx_len;
      for (int i = threadIdx.x; i < HDR; i += CT)
        S.hdr[i] = __ldcg(ctx_t + i);
      __syncthreads();
      mark(0);
      const int m = (int)S.hdr[0];
      const int na = (int)S.hdr[2];
      const int a0m = __ldg(b.mstart + m);
      const bool nspec = t + 1 < A.n && mol_next != m && !bnd &&
                         !(pend && mol_next == m_prev);
      const int var = pend ? acc_prev : 0;  // the partials' outcome set
      const bool margins = S.hdr[3] > 0.0;
      const long long hi_o = order64(S.hdr[81]), lo_o = order64(S.hdr[82]);
      double *part_t = A.part + (size_t)(t % 3) * G * 8;
      constexpr int PF = PART_MAX_GRID / 32;
      if (warp < 4) {
        // warps 0..3 each gather one quantity over the work CTAs (LJ, real
        // space, reciprocal energy, overlap), polling until every CTA's is
        // present; lane l adds CTAs l, l + 32, ... in order, then the warp
        // tree: a fixed order
        const int q = warp;
        constexpr int NPOLL = 3;
        double pp[NPOLL][PF];
        auto issue = [&](double *dst) {
#pragma unroll
          for (int i = 0; i < PF; ++i) {
            int c = lane + 32 * i;
            dst[i] = c < W ? __ldcg(part_t + (size_t)c * 8 + 4 * var + q) : 0.0;
          }
        };
        auto present = [&](const double *src) {
          bool mine = true;
#pragma unroll
          for (int i = 0; i < PF; ++i)
            mine &= __double_as_longlong(src[i]) != (long long)PART_EMPTY;
          return __all_sync(0xffffffffu, mine);
        };
#pragma unroll
        for (int j = 0; j < NPOLL; ++j) {
          if (j)
            __nanosleep(150);
          issue(pp[j]);
        }
        int ok = 1, got = -1;
        unsigned it = 0;
        for (;;) {
#pragma unroll
          for (int j = 0; j < NPOLL; ++j) {
            if (got < 0) {
              if (present(pp[j]))
                got = j;  // warp-uniform
              else
                issue(pp[j]);
            }
          }
          if (got >= 0)
            break;
          int bad = 0;
          if (lane == 0) {
            if (++it > A.spin) {
              atomicOr(b.err, DERR_BARRIER_TIMEOUT);
              bad = 1;
            } else if ((it & 255u) == 0 && *(volatile int *)b.err) {
              bad = 1;
            }
          }
          if (__shfl_sync(0xffffffffu, bad, 0)) {
            ok = 0;
            break;
          }
        }
        if (prof)
          mark(2);
        double pv[PF];
#pragma unroll
        for (int i = 0; i < PF; ++i)
          pv[i] = got == 0 ? pp[0][i] : got == 1 ? pp[1][i] : pp[2][i];
        if (ok) {
          if (q < 3) {
            double v = pv[0];
#pragma unroll
            for (int i = 1; i < PF; ++i)
              if (32 * i < W)  // an FP64 addition takes 64 cycles
                v += pv[i];
            for (int o = 16; o > 0; o >>= 1)
              v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0)
              S.tot[q] = v;
          } else {
            bool any = false;
#pragma unroll
            for (int i = 0; i < PF; ++i)
              any |= __double_as_longlong(pv[i]) != 0;
            any = __any_sync(0xffffffffu, any);
            if (lane == 0)
              S.tot[3] = any ? 1.0 : 0.0;
          }
        }
        if (lane == 0)
          S.red3[0][q] = ok;
        asm volatile("bar.sync 2, 128;" ::: "memory");
        ok = S.red3[0][0] != 0.0 && S.red3[0][1] != 0.0 &&
             S.red3[0][2] != 0.0 && S.red3[0][3] != 0.0;
        int acc = 0;
        if (warp == 0 && ok) {
          double dLJ = 0.0, dRe = 0.0, dRc = 0.0;
          if (lane == 0) {
            const bool over = bits64(S.tot[3]) != 0;
            dLJ = S.tot[0];
            dRe = S.tot[1];
            dRc = (!over && b.K > 0) ? S.tot[2] - S.e_run[2] : 0.0;
            double ex = __dmul_rn(nbeta, __dadd_rn(__dadd_rn(dLJ, dRe), dRc));
            // pacc < exp(ex), decided on logarithms unless the two sides
            // are within 1e-9 (or pacc is 0, or ex not finite); compared as
            // integers of the same order
            const long long xo = order64(ex);
            int res;
            if (margins && xo > hi_o && xo < order64(1.0e300))
              res = 1;
            else if (margins && xo < lo_o && xo > order64(-1.0e300))
              res = 0;
            else
              res = S.hdr[3] < exp(ex);
            acc = res && !over;
            hist = (hist << 1) | (unsigned)acc;
            // what the word releases (coordinates, emptied slots) was
            // fenced at the end of the last move
            st_relaxed(A.seq, dec_word(t, hist));
          }
          acc = __shfl_sync(0xffffffffu, acc, 0);
          if (prof)
            mark(3);
          if (acc) {
            // the new coordinates and centre, after the word (a context
            // built before the next word reads them from its builders'
            // copies of this move)
            if (lane < na) {
              const double *np = S.hdr + 48 + 3 * lane;
              b.x[a0m + lane] = np[0];
              b.y[a0m + lane] = np[1];
              b.z[a0m + lane] = np[2];
            }
            if (lane == 0 && (int)S.hdr[1] == 0) {
              b.cx[m] = S.hdr[4];
              b.cy[m] = S.hdr[5];
              b.cz[m] = S.hdr[6];
            }
          }
          if (lane == 0) {
            if (acc) {
              S.e_run[0] += dLJ;
              S.e_run[1] += dRe;
              S.e_run[2] += dRc;
            }
            if (A.tr_i) {
              A.tr_i[3 * (size_t)t] = (int)S.hdr[1];
              A.tr_i[3 * (size_t)t + 1] = m;
              A.tr_i[3 * (size_t)t + 2] = acc;
              A.tr_d[3 * (size_t)t] = dLJ;
              A.tr_d[3 * (size_t)t + 1] = dRe;
              A.tr_d[3 * (size_t)t + 2] = dRc;
            }
            S.accept = acc;
          }
        }
        if (warp == 0 && lane == 0)
          S.ok = ok;
        // slot set t % 3 of every work CTA, both outcomes, marked empty
        // for move t + 3 (ordered before the next word by the barrier
        // below and that word's release)
        if (ok) {
#pragma unroll
          for (int i = 0; i < PF; ++i) {
            int c = lane + 32 * i;
            if (c < W) {
              __stcg(part_t + (size_t)c * 8 + q, __longlong_as_double(PART_EMPTY));
              __stcg(part_t + (size_t)c * 8 + 4 + q,
                     __longlong_as_double(PART_EMPTY));
            }
          }
        }
      }
      __syncthreads();
      if (!S.ok)
        return;
      const int acc = S.accept;
      if (threadIdx.x == 0) {
        settings_update(S.set, (int)S.hdr[1], acc);
        // releases this CTA's writes with the next word (a release store of
        // the word itself would wait for them then: 0.45 us of every decision)
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
      }
      if (!nspec && t + 1 < A.n) {
        if (!adjust_before(t + 1, bnd))
          return;
        // the next context is built by the work CTAs behind this barrier
        if (!grid_sync(A.bar, G, S.gen, b.err, &S.flag, A.spin))
          return;
      }
      mark(4);
      pend = nspec;
      acc_prev = acc;
      m_prev = m;
    }
  } else {
    // ---------------- work CTAs ----------------
    // warp 7 gathers the next context's inputs, warp 0 counts its writers
    const bool piper = warp == 7 || warp == 0;
    // records and ranges of moves t + 1 and t + 2, the record of t + 3
    CtxPre r1, r2, r3;
    int r1_end = 0, r2_end = 0;
    r1.writer = r2.writer = r3.writer = false;
    r1.m = r2.m = r3.m = -1;
    r1.a0 = r2.a0 = 0;
    if (piper) {
      ctx_pre_record(A, 1, r1);
      ctx_pre_range(A, r1, r1_end);
      ctx_pre_record(A, 2, r2);
      ctx_pre_range(A, r2, r2_end);
      ctx_pre_record(A, 3, r3);
    }
    int nmol2 = A.n > 2 ? A.moves[2].mol : -1;
    bool built1 = false;  // this move's successor has its context already
    bool pend = false;  // this move runs before the previous one's decision
    int m_prev = -1, na_prev = 0;
    int mol_cur = A.n > 0 ? A.moves[0].mol : -1;
    bool have_next = false;  // this move's context prefetched into smem
    // three header buffers in turn: this move's (hc), the previous move's
    // while it is undecided (hq), the next move's, prefetched (hn)
    __shared__ __align__(16) double hbuf[3][HDR];
    int hc = 0, hq = 1, hn = 2;
    for (int t = 0; t < A.n; ++t) {
      const int mol_next = nmol, mol_next2 = nmol2;
      nmol = nmol2;
      nmol2 = t + 3 < A.n ? A.moves[t + 3].mol : -1;
      const bool bnd = adj_r == 0;
      adj_r = adj_r + 1 == S.set.adj ? 0 : adj_r + 1;
      CtxPre pre = r1, pre2 = r2;
      pre.na = r1_end - r1.a0;
      pre2.na = r2_end - r2.a0;
      if (piper) {
        r1 = r2;
        r1_end = r2_end;
        r2 = r3;
        ctx_pre_range(A, r2, r2_end);
        ctx_pre_record(A, t + 4, r3);
      }
      // ---------------- phase A ----------------
      const double *ctx_t = A.ctx + (size_t)(t % PIPE_NCTX) * A.ctx_len;
      const int m = mol_cur;
      // this move's atom count, from the record pipeline of warp 0 (stored
      // during the previous move) but for the first move
      __shared__ int nx_na;
      const int na = t == 0 ? __ldg(b.mstart + m + 1) - __ldg(b.mstart + m)
                            : nx_na;
      // may move t + 1 run before this move's decision
      const bool nspec = t + 1 < A.n && mol_next != m && !bnd &&
                         !(pend && mol_next == m_prev);
      // A context takes longer to write and reach every CTA than the rest of
      // a phase (9,200 of 15,900 cycles on 256 waters), so that of move t + 2
      // is written during this phase where it can be: its molecule is none of
      // those that move or may have moved meanwhile, and no settings
      // adjustment precedes it or move t + 1.  Else it is written during
      // phase A(t + 1), as that of t + 1 is now if it was not yet.
      const bool early2 = nspec && t + 2 < A.n && adj_r != 0 &&
                          mol_next2 != m && mol_next2 != mol_next &&
                          !(pend && mol_next2 == m_prev);
      const bool late1 = nspec && !built1;
      pre.writer = pre2.writer = false;
      const bool wload = late1 && warp == 7, wload2 = early2 && warp == 7;
      const int nbuild = max(1, min(W, b.K > 0 ? 2 * pre.na * 3 : 0));
      double lj = 0.0, re = 0.0, ovl = 0.0, er = 0.0, er2 = 0.0;
      // pair terms of the previous move's atoms this CTA owns, at their
      // old positions (that move rejected) and new ones (accepted)
      double ljR = 0.0, reR = 0.0, ovR = 0.0, ljA = 0.0, reA = 0.0, ovA = 0.0;
      // this move's new sums on either outcome of the previous move
      int fr[3], nfr = 0;
      for (int i = 0; i < 4; ++i)
        if (i != bS && i != bP && nfr < 3)
          fr[nfr++] = i;
      const int bR = fr[0], bA = fr[1];
      // Real space, as in k_chain_fp64: own atoms against the old and new
      // positions of the moved atoms, FP32 pre-test on fixed-point turns,
      // the pairs compacted in order into a shared list.  While the previous
      // move is undecided, its atoms are left out of the pre-test and listed
      // after the others on both of its outcomes, so that one warp pass
      // takes them all.
      __shared__ double2 icl_pos[ICL_CAP][2];
      __shared__ int icl_meta[ICL_CAP];
      // position (old atoms, then new) | class << 8 | turn_wrap << 16; class 0
      // an own atom that both outcomes of the previous move share, 1 / 2 an
      // atom of the previous move's molecule at its old position (that move
      // rejected) / its new one (accepted)
      __shared__ int icl_tag[ICL_CAP];
      __shared__ int seg_cnt[PNSEG];  // entries found per segment
      const int npos = 2 * na;
      double *const hd = hbuf[hc];        // this move's header
      const double *const hdrp = hbuf[hq];  // the previous move's
      const uint32_t *pturn = (const uint32_t *)(hd + 84);
      // own atoms of the previous molecule (usually 0 or 1)
      const int2 *const ownp = (const int2 *)(hdrp + 120);
      int n_prev = 0;
      if (pend && !kless)
        for (int ap = 0; ap < na_prev; ++ap)
          n_prev += ownp[ap].x == orank;
      const int ncomb = n_prev * 2 * npos;
      double *const part_c = A.part + (size_t)(t % 3) * G * 8 + (size_t)cta * 8;
      // Lists, from slot n on and below slot lim, the pairs of 32 own atoms
      // (one a lane) with this move's positions p0, p0 + step, ...: an FP32
      // pre-test of them all, then for each position that some lane passes a
      // ballot that gives the lanes their slots.  Pairs past lim are
      // evaluated here (not met at liquid densities).  Returns the end of
      // the entries.
      auto list_own = [&](int i, bool valid, int p0, int step, int n,
                          int lim) -> int {
        uint4 f = make_uint4(0, 0, 0, 0);
        double2 pxy = make_double2(0.0, 0.0), pzq = pxy;
        unsigned hit = 0;  // bit p: position p passes the pre-test
        if (valid) {
          f = ot[i];
          pxy = oxy[i];
          pzq = ozq[i];
          const int mj = meta_mol((int)f.w);
          if (mj != m && !(pend && mj == m_prev))
#pragma unroll 2
            for (int pp = p0; pp < npos; pp += step) {
              float dx = (float)(int)(pturn[3 * pp] - f.x) * turn_f[0];
              float dy = (float)(int)(pturn[3 * pp + 1] - f.y) * turn_f[1];
              float dz = (float)(int)(pturn[3 * pp + 2] - f.z) * turn_f[2];
              if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cut_f)
                hit |= 1u << pp;
            }
        }
        for (unsigned any = __reduce_or_sync(0xffffffffu, hit); any;
             any &= any - 1) {
          const int pp = __ffs(any) - 1;
          const bool mine = hit >> pp & 1;
          const unsigned mask = __ballot_sync(0xffffffffu, mine);
          const int pos = n + __popc(mask & ((1u << lane) - 1));
          n += __popc(mask);
          const unsigned wr = turn_wrap(pturn + 3 * pp, f);
          if (mine && pos < lim) {
            icl_pos[pos][0] = pxy;
            icl_pos[pos][1] = pzq;
            icl_meta[pos] = (int)f.w;
            icl_tag[pos] = pp | (int)wr << 16;
          } else if (mine) {
            const int side = pp >= na;
            pair_term_pipe(A, hd, pp - side * na, side, pxy, pzq, (int)f.w, wr,
                           lj12, coul_cut, ptab, lj, re, ovl);
          }
        }
        return n;
      };
      // The previous move's atoms this CTA owns on both outcomes (entries
      // c = (atom, outcome, position)), pre-tested like the others and
      // appended in order from slot n0 by one warp, below slot lim; those
      // past it are evaluated here.  Returns the end of the entries.
      auto list_prev = [&](int n0, int lim) -> int {
        int n = n0;
        const int nc = na_prev * 2 * npos;
        for (int base = 0; base < nc; base += 32) {
          const int c = base + lane;
          bool hit = false;
          int i = 0, vr = 0, ap = 0, pp = 0;
          uint4 f = make_uint4(0, 0, 0, 0);
          if (c < nc) {
            ap = c / (2 * npos);
            const int r = c - ap * 2 * npos;
            vr = r / npos;
            pp = r - vr * npos;
            if (ownp[ap].x == orank) {
              i = ownp[ap].y;
              f = ot[i];
              if (vr) {
                const uint32_t *nt = (const uint32_t *)(hdrp + 84) + (na_prev + ap) * 3;
                f.x = nt[0];
                f.y = nt[1];
                f.z = nt[2];
              }
              float dx = (float)(int)(pturn[3 * pp] - f.x) * turn_f[0];
              float dy = (float)(int)(pturn[3 * pp + 1] - f.y) * turn_f[1];
              float dz = (float)(int)(pturn[3 * pp + 2] - f.z) * turn_f[2];
              hit = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cut_f;
            }
          }
          const unsigned mask = __ballot_sync(0xffffffffu, hit);
          if (hit) {
            const int pos = n + __popc(mask & ((1u << lane) - 1));
            const int side = pp >= na ? 1 : 0, a = pp - side * na;
            double2 pxy = oxy[i], pzq = ozq[i];
            if (vr) {
              const double *np = hdrp + 48 + 3 * ap;
              pxy = make_double2(np[0], np[1]);
              pzq.x = np[2];
            }
            const unsigned wr = turn_wrap(pturn + 3 * pp, f);
            if (pos < lim) {
              icl_pos[pos][0] = pxy;
              icl_pos[pos][1] = pzq;
              icl_meta[pos] = (int)f.w;
              icl_tag[pos] = pp | (1 + vr) << 8 | (int)wr << 16;
            } else {
              pair_term_pipe(A, hd, a, side, pxy, pzq, (int)f.w, wr, lj12,
                             coul_cut, ptab, vr ? ljA : ljR, vr ? reA : reR,
                             vr ? ovA : ovR);
            }
          }
          n += __popc(mask);
        }
        return n;
      };
      // the listed pairs, by the lanes of one warp, each added to its
      // class's sums (the v-th listed entry counting through the segments
      // in order)
      double psum[4];  // LJ and real space, previous move rejected, accepted
      bool ov0, ov1;
      auto eval_pairs = [&](int n_eval, int nseg) {
        psum[0] = psum[1] = psum[2] = psum[3] = 0.0;
        ov0 = ov1 = false;
        for (int v = lane; v < n_eval; v += 32) {
          int i = v, before = 0;
#pragma unroll
          for (int sg = 0; sg < PNSEG; ++sg)
            if (sg < nseg) {
              if (v >= before)
                i = sg * PSEG + v - before;
              before += min(seg_cnt[sg], PSEG);
            }
          double e, l;
          bool o;
          const int tag = icl_tag[i], pp = tag & 255, side = pp >= na;
          if (!pair_energy_pipe(A, hd, pp - side * na, side, icl_pos[i][0],
                                icl_pos[i][1], icl_meta[i], (unsigned)tag >> 16,
                                lj12, coul_cut, ptab, e, l, o))
            continue;
          const int c = tag >> 8 & 255;
          const double t4[4] = {c == 2 ? 0.0 : l, c == 2 ? 0.0 : e,
                                c == 1 ? 0.0 : l, c == 1 ? 0.0 : e};
          ov0 |= o && c != 2;
          ov1 |= o && c != 1;
          if (v == lane) {  // a lane's first pair: no additions
            for (int j = 0; j < 4; ++j)
              psum[j] = t4[j];
          } else {
            for (int j = 0; j < 4; ++j)
              psum[j] += t4[j];
          }
        }
      };
      // the pair partials of the warp that evaluated this CTA's pairs: warp
      // sums on both outcomes, into slots 0, 1 and 4, 5
      auto store_pairs_warp = [&]() {
        const bool any0 = __any_sync(0xffffffffu, ov0),
                   any1 = __any_sync(0xffffffffu, ov1);
        if (ncomb > 0) {
          const double v = warp_sum4(psum);
          if ((lane & 7) == 0)
            __stcg(part_c + (lane >> 3 & 1) + 4 * (lane >> 4), v);
        } else {
          // both outcomes share every pair of this CTA
          const double v = warp_sum2(psum[0], psum[1]);
          if ((lane & 15) == 0) {
            __stcg(part_c + (lane >> 4), v);
            __stcg(part_c + 4 + (lane >> 4), v);
          }
        }
        if (lane == 0) {
          __stcg(part_c + 3, any0 ? 1.0 : 0.0);
          __stcg(part_c + 7, any1 ? 1.0 : 0.0);
        }
      };

      // What this CTA waits for before its next phase A, polled by one warp
      // that is otherwise idle (its loads' round trips hidden behind the
      // phase): the previous move's decision and the flags of the next
      // context's writers when the next move runs ahead, else this move's
      // decision.  The decision word (lane 0) until it has passed move
      // `want`; S.ok false when a wait gave up.
      const int want = nspec ? (pend ? t - 1 : -1) : t;
      auto poll_warp = [&]() {
        unsigned w = 0;
        int ok = 1;
        // the flags by relaxed loads and one fence once all are seen; the
        // word, which the CTA waits for, by acquire loads (a fence after it
        // came would cost about as long as a load)
        auto wait_for = [&](auto seen) {
          for (unsigned it = 0; ok;) {
            if (__all_sync(0xffffffffu, seen()))
              break;
            int bad = 0;
            if (lane == 0) {
              if (++it > A.spin) {
                atomicOr(b.err, DERR_BARRIER_TIMEOUT);
                bad = 1;
              } else if ((it & 255u) == 0 && *(volatile int *)b.err) {
                bad = 1;
              }
            }
            if (__shfl_sync(0xffffffffu, bad, 0))
              ok = 0;
            __nanosleep(32);
          }
        };
        if (nspec) {
          wait_for([&]() {
            bool mine = true;
            for (int c = lane; c < nbuild; c += 32)
              mine &= (int)(ld_relaxed(A.seq + SEQ_CTX + c) - (unsigned)(t + 1)) >= 0;
            return mine;
          });
          asm volatile("fence.acq_rel.gpu;" ::: "memory");
          if (ok && !kless) {
            // the next context is complete: its header and phase rows into
            // shared memory now, off the next phase A's path, eight loads in
            // flight a lane
            const double2 *src =
                (const double2 *)(A.ctx + (size_t)((t + 1) % PIPE_NCTX) * A.ctx_len);
            double2 *tabn = tab == tab0 ? tab1 : tab0;
            double2 *hn2 = (double2 *)hbuf[hn];
            const int nh = HDR / 2, n = nh + A.nrows_max * stride;
            for (int i0 = lane; i0 < n; i0 += 8 * 32) {
              double2 v[8];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (i0 + 32 * j < n)
                  v[j] = __ldcg(src + i0 + 32 * j);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int i = i0 + 32 * j;
                if (i < nh)
                  hn2[i] = v[j];
                else if (i < n)
                  tabn[i - nh] = v[j];
              }
            }
          }
        }
        if (want >= 0)
          wait_for([&]() {
            if (lane == 0)
              w = ld_acquire(A.seq);
            return lane != 0 || (int)(w >> 4) >= want + 1;
          });
        if (lane == 0) {
          S.ok = ok && *(volatile int *)b.err == 0;
          S.word = w;
        }
      };

      if (kless) {
        // A context writer without k-vectors and atoms.  Warp 0 takes this
        // move's header and stores empty partials; warps 1..7 write their
        // part of a coming move's context meanwhile, from the start of the
        // phase (it does not depend on this move's header).
        if (warp == 0) {
          for (int i = lane; i < HDR; i += 32)
            hd[i] = __ldcg(ctx_t + i);
          __syncwarp();
          mark(0);
          mark(1);
          if (lane < 8)  // no k-vectors and no atoms: nothing to add
            __stcg(part_c + lane, 0.0);
          poll_warp();
        } else if (nspec) {
          auto build = [&](int s, CtxPre &c) {
            if (warp == 7) {
              ctx_pre2(A, S, s, c);
              if (c.writer)
                ctx_pre_store(S, c);
              if (lane == 0)
                S.b_writer = c.writer;
            }
            group_sync(CT - 32);
            if (S.b_writer) {
              build_ctx_rest(A, S, s, (int)threadIdx.x - 32, CT - 32);
              group_sync(CT - 32);
              if (threadIdx.x == 32)
                st_release(A.seq + SEQ_CTX + blockIdx.x, (unsigned)s);
            }
          };
          if (late1)
            build(t + 1, pre);
          if (early2) {
            if (late1)
              group_sync(CT - 32);  // S.b_* read before they change
            build(t + 2, pre2);
          }
        }
        __syncthreads();
        mark(2);
      } else {
        // A CTA with a k-chunk.  Warp 3 evaluates the listed pairs beside
        // the k-vectors of warps 0, 1, 2, 4, 5, 6 (warps issue to the SM's
        // sub-partitions by index modulo 4); each stores its partials as
        // soon as they are summed.  Warp 7 of a context writer with
        // k-vectors builds its part of the next context.
        if (have_next) {
          // header and rows prefetched by the polling warp during the
          // previous phase A (behind that phase's closing barriers)
          tab = tab == tab0 ? tab1 : tab0;
        } else {
          for (int i = threadIdx.x; i < HDR; i += CT)
            hd[i] = __ldcg(ctx_t + i);
          for (int i = threadIdx.x; i < A.nrows_max * stride; i += CT)
            tab[i] = __ldcg((const double2 *)(ctx_t + HDR) + i);
          __syncthreads();
        }
        mark(0);
        if (wload)
          ctx_pre2(A, S, t + 1, pre);
        else if (wload2)
          ctx_pre2(A, S, t + 2, pre2);
        // warps 0-6 list the pairs of 32 own atoms at a time with all
        // positions (with a share of them where there are fewer such blocks
        // than warps), each into its own segment; warp 7 forms the x-y
        // column products and lists the previous move's atoms into the last
        if (warp < 7) {
          int n = warp * PSEG;
          const int nb = (on + 31) / 32;
          const int share = nb > 3 ? 1 : min(npos, 7 / max(nb, 1));
          for (int u = warp; u < nb * share; u += 7) {
            const int p0 = share > 1 ? u / nb : 0, i = (u - p0 * nb) * 32 + lane;
            n = list_own(i, i < on, p0, share, n, (warp + 1) * PSEG);
          }
          if (lane == 0)
            seg_cnt[warp] = n - warp * PSEG;
        } else {
          xy_products(lane, 32, npair, pair_n, tab, stride, na, hd + 72, exy);
          const int b0 = 7 * PSEG;
          const int n = ncomb > 0 ? list_prev(b0, ICL_CAP) - b0 : 0;
          if (lane == 0)
            seg_cnt[7] = n;
        }
        __syncthreads();  // the listed pairs
        mark(1);
        // pairs past a full segment were evaluated where they were found
        // (not met at liquid densities): then the pair sums are the CTA's
        int n_eval = 0;
        bool all_pairs = false;
        for (int sg = 0; sg < PNSEG; ++sg) {
          n_eval += min(seg_cnt[sg], PSEG);
          all_pairs |= seg_cnt[sg] > PSEG;
        }
        if (warp == pw) {
          eval_pairs(n_eval, PNSEG);
          if (!all_pairs)
            store_pairs_warp();
        } else if (warp == 7) {
          if (wload && pre.writer) {
            ctx_pre_store(S, pre);
            __syncwarp();
            build_ctx_warp(A, S, t + 1);
          }
          if (wload2) {
            if (wload)
              ctx_pre2(A, S, t + 2, pre2);
            if (pre2.writer) {
              __syncwarp();
              ctx_pre_store(S, pre2);
              __syncwarp();
              build_ctx_warp(A, S, t + 2);
            }
          }
          if (!all_pairs)
            poll_warp();
        } else {
          const int kw = warp < 3 ? warp : warp - 1;  // 0..5
          const double *sR = KR(bS), *sI = KI(bS);
          const double *pR = pend ? KR(bP) : nullptr;
          const double *pI = pend ? KI(bP) : nullptr;
          double *rR = KR(bR), *rI = KI(bR), *aR = KR(bA), *aI = KI(bA);
          for (int i = kw * 32 + lane; i < kc; i += 6 * 32) {
            double dR, dI;
            kvec_delta(kn[i],
                       npair > 0 ? exy + (size_t)pidx[i] * 2 * na : nullptr,
                       tab, stride, na, hd + 72, dR, dI);
            double srn = sR[i] + dR, sin_ = sI[i] + dI;
            rR[i] = srn;
            rI[i] = sin_;
            er += (srn * srn + sin_ * sin_) * pf[i];
            if (pend) {
              double arn = pR[i] + dR, ain = pI[i] + dI;
              aR[i] = arn;
              aI[i] = ain;
              er2 += (arn * arn + ain * ain) * pf[i];
            }
          }
          // the reciprocal energy of the chunk on both outcomes: warp sums,
          // then the six warps in order (named barrier 4)
          const double ew = warp_sum2(er, er2);
          if ((lane & 15) == 0)
            red6[lane ? 5 : 2][warp] = ew;
          asm volatile("bar.sync 4, 192;" ::: "memory");
          if (warp == 0) {
            // lanes 0-7 the six warps' er, lanes 8-15 their er2
            const int w = lane & 7;
            double r = lane < 16 && w != 3 && w != 7 ? red6[lane < 8 ? 2 : 5][w] : 0.0;
            for (int o = 4; o > 0; o >>= 1)
              r += __shfl_xor_sync(0xffffffffu, r, o);
            if (lane == 0) {
              __stcg(part_c + 2, r);
              if (!pend)
                __stcg(part_c + 6, r);
            } else if (lane == 8 && pend) {
              __stcg(part_c + 6, r);
            }
          }
        }
        if (all_pairs) {
          // pairs past the list were evaluated by every warp: the CTA's
          // pair sums over all warps, in warp order
          double v[4] = {lj + ljR, re + reR, lj + ljA, re + reA};
          if (warp == pw)
            for (int j = 0; j < 4; ++j)
              v[j] += psum[j];
          for (int o = 16; o > 0; o >>= 1)
            for (int j = 0; j < 4; ++j)
              v[j] += __shfl_down_sync(0xffffffffu, v[j], o);
          const bool mine = warp == pw;
          const int any0 = __syncthreads_or(ovl > 0.0 || ovR > 0.0 || (mine && ov0));
          const int any1 = __syncthreads_or(ovl > 0.0 || ovA > 0.0 || (mine && ov1));
          if (lane == 0) {
            red6[0][warp] = v[0];
            red6[1][warp] = v[1];
            red6[3][warp] = v[2];
            red6[4][warp] = v[3];
          }
          __syncthreads();
          if (threadIdx.x < 4) {
            const int j = threadIdx.x < 2 ? threadIdx.x : threadIdx.x + 1;
            double r = 0.0;
            for (int w = 0; w < CT / 32; ++w)
              r += red6[j][w];
            __stcg(part_c + (threadIdx.x < 2 ? threadIdx.x : threadIdx.x + 2), r);
          } else if (threadIdx.x == 4) {
            __stcg(part_c + 3, any0 ? 1.0 : 0.0);
            __stcg(part_c + 7, any1 ? 1.0 : 0.0);
          }
          // the poll after the CTA-wide sums (warp 7 took part in them)
          if (warp == 7)
            poll_warp();
        }
        __syncthreads();
        mark(2);
      }
      // ---------------- phase B ----------------
      // an accepted move (hd: its header): its new positions for the next
      // contexts, and the moved atoms this CTA owns take them
      auto commit_atoms = [&](const double *hd, int nn) {
        for (int i = threadIdx.x; i < 3 * nn + 3; i += CT) {
          if (i < 3 * nn)
            S.last_newp[i / 3][i % 3] = hd[48 + i];
          else
            S.last_newcom[i - 3 * nn] = hd[4 + i - 3 * nn];
        }
        for (int a = threadIdx.x; a < nn; a += CT) {
          const int2 ow = ((const int2 *)(hd + 120))[a];
          if (ow.x == orank) {
            const int i = ow.y;
            const double *np = hd + 48 + 3 * a;
            const uint32_t *pt = (const uint32_t *)(hd + 84) + (nn + a) * 3;
            oxy[i] = make_double2(np[0], np[1]);
            ozq[i].x = np[2];
            ot[i] = make_uint4(pt[0], pt[1], pt[2], ot[i].w);
          }
        }
      };
      if (!S.ok)
        return;
      const unsigned word = S.word;
      if (threadIdx.x == 0)  // the next move's count (read after a barrier)
        nx_na = pre.na;
      if (pend) {
        const int acc_p = dec_outcome(word, t - 1);
        if (threadIdx.x == 0) {
          settings_update(S.set, (int)hdrp[1], acc_p);
          S.last_m = m_prev;
          S.last_acc = acc_p;
        }
        if (acc_p) {
          commit_atoms(hdrp, na_prev);
          bS = bP;  // the previous move's new sums are committed
          bP = bA;  // and this move's new sums on that outcome pend
        } else {
          bP = bR;
        }
        __syncthreads();  // the previous header is read before it is replaced
      } else {
        bP = bR;
      }
      mark(3);
      if (nspec) {
        m_prev = m;
        na_prev = na;
        pend = true;
        have_next = !kless;
        __syncthreads();
      } else {
        // this move's decision and commit, then the next context behind a
        // grid barrier
        const int acc = dec_outcome(word, t);
        __syncthreads();
        if (threadIdx.x == 0) {
          settings_update(S.set, (int)hd[1], acc);
          S.last_m = m;
          S.last_acc = acc;
        }
        if (acc) {
          commit_atoms(hd, na);
          bS = bP;
        }
        bP = -1;
        have_next = false;
        __syncthreads();
        if (t + 1 < A.n) {
          if (!adjust_before(t + 1, bnd))
            return;
          build_ctx(A, S, t + 1, hd, acc, 0, CT);
          if (!grid_sync(A.bar, G, S.gen, b.err, &S.flag, A.spin))
            return;
        }
        pend = false;
      }
      mark(4);
      mol_cur = mol_next;
      built1 = early2;
      // the headers' roles: this move's becomes the previous one's, the
      // prefetched one (or a free buffer) this move's
      const int hfree = hq;
      hq = hc;
      hc = hn;
      hn = hfree;
    }
  }
  if (prof) {
    for (int ph = 0; ph < 5; ++ph)
      A.prof[5 * pslot + ph] += pacc[ph];
    A.prof[10 + pslot] += A.n;
  }
  // write back this CTA's structure factors; the decider the settings and
  // the running energies
  for (int i = threadIdx.x; i < kc; i += CT) {
    b.sumRref[kbeg + i] = KR(bS)[i];
    b.sumIref[kbeg + i] = KI(bS)[i];
  }
  if (leader && threadIdx.x == 0) {
    *A.set = S.set;
    for (int i = 0; i < 5; ++i)
      b.energy[i] = S.e_run[i];
  }
}
