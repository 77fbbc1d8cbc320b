// Ewald reciprocal-space kernels (FP64 plain form).
//
//   energy            sum_k prefact_k (sumR^2 + sumI^2)
//                     (Ewald::BoxReciprocal, src/Ewald.cpp:375-406)
//   molecule delta    sumNew = sumRef + new - old, energy difference
//                     (Ewald::MolReciprocal, src/Ewald.cpp:409-473) and the
//                     insert / delete deltas (SwapDestRecip / SwapSourceRecip,
//                     src/Ewald.cpp:478-531, 657-710)
//   reciprocal force  (Ewald::BoxForceReciprocal, src/Ewald.cpp:1496-1596)
//
// The sums over all atoms and k-vectors are in gb_ewald.cu.
#include "gb_box.h"
#include "gb_fixed.cuh"
#include "gb_pair.cuh"

namespace gb {

// ---------------------------------------------------------------------------
// Energy of a set of structure factors
// ---------------------------------------------------------------------------
constexpr int ET = 256;
__global__ void k_recip_energy(DevBox b, const double *__restrict__ sR,
                               const double *__restrict__ sI, double *part) {
  int k = blockIdx.x * ET + threadIdx.x;
  double e = 0.0;
  if (k < b.K)
    e = ((sR[k] * sR[k] + sI[k] * sI[k]) * b.prefact[k]);
  __shared__ double red[ET / 32];
  double s = block_sum<ET>(e, red);
  if (threadIdx.x == 0)
    part[blockIdx.x] = s;
}

__global__ void k_sum_in_order(const double *__restrict__ part, int n,
                               const double *sub, double *out) {
  __shared__ double red[ET / 32];
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += ET)
    v += part[i];
  double s = block_sum<ET>(v, red);
  if (threadIdx.x == 0)
    out[0] = sub ? s - sub[0] : s;
}

int launch_recip_energy(Box &bx, const double *sumR, const double *sumI,
                        double *d_out) {
  return launch_recip_energy_view(bx, bx.dev, sumR, sumI, d_out);
}

// The energy of sums with the prefactors and k count of a view (the New
// k-vector set for a trial volume).
int launch_recip_energy_view(Box &bx, const DevBox &b, const double *sumR,
                             const double *sumI, double *d_out) {
  int nb = (b.K + ET - 1) / ET;
  int rc = bx.EnsureScratch(nb);
  if (rc)
    return rc;
  k_recip_energy<<<nb, ET, 0, bx.stream>>>(b, sumR, sumI, bx.d_scratch);
  k_sum_in_order<<<1, ET, 0, bx.stream>>>(bx.d_scratch, nb, nullptr, d_out);
  return bx.CudaCheck(cudaGetLastError(), "recip energy");
}

// ---------------------------------------------------------------------------
// One-molecule delta.  mode 0: displacement/rotation (new - old),
// 1: insertion (+ new), 2: deletion (- given positions).  One launch: every
// CTA forms the phase rows exp(i n 2 pi r_d / L_d) of up to eight positions at
// a time in fixed point (integer work; the sine and cosine of every k . r in
// FP64 cost about 100 instructions of 64 cycles each), a thread then sums its
// k-vector's products, and the last CTA adds the energies.
// ---------------------------------------------------------------------------
constexpr int MRT = 128;  // threads (k-vectors) per CTA
constexpr int MRP = 8;    // positions per pass
template <int N>
struct NewPos {
  double xyz[3 * N];
};

template <int N>
__global__ void __launch_bounds__(MRT) k_mol_recip(DevBox b, int m,
                                                   const __grid_constant__ NewPos<N> P,
                                                   int mode, double *part,
                                                   double *out) {
  extern __shared__ double2 rows[];  // [MRP][3][kmax + 1]
  __shared__ unsigned long long us[3 * MRP];
  __shared__ double qs[MRP];
  __shared__ int bad;  // a coordinate that is not finite
  const int k = blockIdx.x * MRT + threadIdx.x;
  const int stride = b.kmax + 1;
  const int a0 = b.mstart[m], n = b.mstart[m + 1] - a0;
  const int np = mode == 0 ? 2 * n : n;  // new positions, then the old ones
  char4 kn = make_char4(0, 0, 0, 0);
  if (k < b.K)
    kn = b.kn[k];
  if (threadIdx.x == 0)
    bad = 0;
  double dR = 0.0, dI = 0.0;
  for (int p0 = 0; p0 < np; p0 += MRP) {
    const int cnt = min(MRP, np - p0);
    __syncthreads();
    if (threadIdx.x < 3 * cnt) {
      const int p = p0 + threadIdx.x / 3, d = threadIdx.x % 3;
      const int a = a0 + (p < n ? p : p - n);
      const double x = p < n ? P.xyz[3 * p + d]
                             : (d == 0 ? b.x : d == 1 ? b.y : b.z)[a];
      us[threadIdx.x] = turn64(x, b.L[d]);
      if (!isfinite(x))
        bad = 1;
      if (d == 0) {
        const double q = b.q[a];
        // - for the old positions and for a deletion
        qs[threadIdx.x / 3] = fabs(q) < 0.000000001      ? 0.0
                              : (p >= n || mode == 2) ? -q
                                                      : q;
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * cnt * stride; e += MRT) {
      const int r = e / stride, j = e - r * stride;
      const Cis c = cis_q62(us[r] * (unsigned long long)j);
      const double f = (r % 3 ? 1.0 : qs[r / 3]) / 4611686018427387904.0;  // 2^62
      rows[e] = make_double2((double)c.c * f, (double)c.s * f);
    }
    __syncthreads();
    for (int p = 0; p < cnt; ++p) {
      const double2 *r = rows + (size_t)(3 * p) * stride;
      const double2 x = r[kn.x];
      double2 y = r[stride + abs(kn.y)], z = r[2 * stride + abs(kn.z)];
      if (kn.y < 0)
        y.y = -y.y;
      if (kn.z < 0)
        z.y = -z.y;
      const double2 v = make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
      dR = fma(v.x, z.x, fma(-v.y, z.y, dR));
      dI = fma(v.x, z.y, fma(v.y, z.x, dI));
    }
  }
  double e = 0.0;
  if (k < b.K) {
    if (bad)
      dR = dI = nan("");
    const double sr = b.sumRref[k] + dR, si = b.sumIref[k] + dI;
    b.sumRnew[k] = sr;
    b.sumInew[k] = si;
    e = (sr * sr + si * si) * b.prefact[k];
  }
  // The energy in the order of k_recip_energy and k_sum_in_order (the sums of
  // 256 k-vectors as eight warp sums in turn, these over 256 threads), so
  // that the rounding of the new and the stored energy cancels in their
  // difference.
  for (int o = 16; o > 0; o >>= 1)
    e += __shfl_down_sync(0xffffffffu, e, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    part[blockIdx.x * (MRT / 32) + warp] = e;
  if (!last_cta((unsigned *)b.err + 2))
    return;
  __shared__ double red[ET / 32];
  const int nw = gridDim.x * (MRT / 32), nb = (b.K + ET - 1) / ET;
  for (int vw = warp; vw < ET / 32; vw += MRT / 32) {
    double v = 0.0;
    for (int i = vw * 32 + lane; i < nb; i += ET) {
      double c = 0.0;
      for (int w = 0; w < ET / 32; ++w)
        if (i * (ET / 32) + w < nw)
          c += __ldcg(part + i * (ET / 32) + w);
      v += c;
    }
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0)
      red[vw] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
    for (int w = 0; w < ET / 32; ++w)
      v += red[w];
    out[0] = v - b.energy[2];  // - sysPotRef.boxEnergy[box].recip
  }
}

template <int N>
static int launch_mol_recip_n(Box &bx, int m, const double *newpos, int n,
                              int mode) {
  const DevBox &b = bx.dev;
  const int nb = (b.K + MRT - 1) / MRT;
  int rc = bx.EnsureScratch((size_t)nb * (MRT / 32));
  if (rc)
    return rc;
  NewPos<N> P;
  for (int i = 0; i < 3 * n; ++i)
    P.xyz[i] = newpos[i];
  const size_t sh = (size_t)3 * MRP * (b.kmax + 1) * sizeof(double2);
  raise_smem_limit((const void *)k_mol_recip<N>, sh);
  k_mol_recip<N><<<nb, MRT, sh, bx.stream>>>(b, m, P, mode, bx.d_scratch,
                                             bx.h_pinned);
  return bx.CudaCheck(cudaGetLastError(), "mol recip");
}

int launch_mol_recip(Box &bx, int m, const double *newpos, int mode) {
  const int n = bx.host.mstart[m + 1] - bx.host.mstart[m];
  return n <= 16 ? launch_mol_recip_n<16>(bx, m, newpos, n, mode)
                 : launch_mol_recip_n<64>(bx, m, newpos, n, mode);
}

// ---------------------------------------------------------------------------
// Reciprocal forces: the k-space part (gb_ewald.cu) and, per atom, the
// intramolecular correction (src/Ewald.cpp:1556-1575).
// ---------------------------------------------------------------------------
// (erf(a r) / r - 2 a / sqrt(pi) exp(-a^2 r^2)) / r^2.  The two terms nearly
// cancel inside a molecule (a r below one: 30-fold at 1 A), so there their
// difference is summed as its own series,
//   a^3 (4 / sqrt(pi)) sum_j (-u)^j / (j! (2 j + 3)),  u = a^2 r^2,
// to j = 17 (the next term is below 1e-17 of the sum for u <= 1): 18
// multiply-adds and no erf, exp, root or division.
__device__ __forceinline__ double intra_factor(const FF &ff, double distSq) {
  const double u = ff.alphaSq * distSq;
  if (u <= 1.0) {
    constexpr double INV_FACT[18] = {
        1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720,
        1.0 / 5040, 1.0 / 40320, 1.0 / 362880, 1.0 / 3628800,
        1.0 / 39916800, 1.0 / 479001600, 1.0 / 6227020800.0,
        1.0 / 87178291200.0, 1.0 / 1307674368000.0, 1.0 / 20922789888000.0,
        1.0 / 355687428096000.0};
    double p = 0.0;
#pragma unroll
    for (int j = 17; j >= 0; --j)
      p = fma(p, -u, INV_FACT[j] / (2 * j + 3));
    return ff.alpha * ff.alphaSq * (2.0 * M_2_SQRTPI) * p;
  }
  const double dist = sqrt(distSq);
  return (erf(ff.alpha * dist) / dist -
          ff.alpha * M_2_SQRTPI * exp(-1.0 * ff.alphaSq * distSq)) / distSq;
}

__global__ void __launch_bounds__(128) k_force_recip(DevBox b, const FF *__restrict__ pff,
                                                     const double *__restrict__ fpart,
                                                     int nfp, double *aR) {
  const FF &ff = *pff;
  const int a = blockIdx.x * 128 + threadIdx.x;
  if (a >= b.n_atoms)
    return;
  double f[3] = {0.0, 0.0, 0.0};
  for (int c = 0; c < nfp; ++c)
    for (int d = 0; d < 3; ++d)
      f[d] += fpart[((size_t)c * 3 + d) * b.n_atoms + a];
  const double q = b.q[a];
  if (fabs(q) >= 0.000000001) {
    const int m = b.mol[a];
    for (int j = b.mstart[m]; j < b.mstart[m + 1]; j++) {
      if (j == a)
        continue;
      double dx = min_image(b.x[a] - b.x[j], b.L[0], b.half[0]);
      double dy = min_image(b.y[a] - b.y[j], b.L[1], b.half[1]);
      double dz = min_image(b.z[a] - b.z[j], b.L[2], b.half[2]);
      const double g = q * b.q[j] * QQ_FACT * intra_factor(ff, dsq3(dx, dy, dz));
      f[0] -= g * dx;
      f[1] -= g * dy;
      f[2] -= g * dz;
    }
  }
  for (int d = 0; d < 3; ++d)
    aR[3 * (size_t)a + d] = f[d];
}

int launch_force_recip(Box &bx, const DevBox &b, const double *sumR,
                       const double *sumI, double *aR, double *mR) {
  if (!bx.cfg.ewald) {
    cudaMemsetAsync(aR, 0, (size_t)b.n_atoms * 24, bx.stream);
    cudaMemsetAsync(mR, 0, (size_t)b.n_mol * 24, bx.stream);
    return bx.CudaCheck(cudaGetLastError(), "force recip");
  }
  double *fpart, *none;
  int nfp;
  int rc = launch_force_split(bx, b, sumR, sumI, 0, &fpart, &nfp, &none);
  if (rc)
    return rc;
  k_force_recip<<<(b.n_atoms + 127) / 128, 128, 0, bx.stream>>>(b, bx.d_ff,
                                                                fpart, nfp, aR);
  return launch_mol_force(bx, b, aR, mR);
}

}  // namespace gb

namespace gb {

// ---------------------------------------------------------------------------
// Reciprocal virial (Ewald::VirialReciprocal, src/Ewald.cpp:1168-1305) from
// the Ref structure factors: the k-space sum, one thread per k-vector,
//   w_d += prefact |S|^2 (1 - 2 (1/(4 alpha^2) + 1/k^2) k_d^2),
// and the intramolecular part, one thread per atom,
//   w_d += -F_d (r_d - com_d),
// F the reciprocal force of the atom without the intramolecular correction
// (launch_force_split): sum_k 2 q prefact (S_I cos - S_R sin) k_d
// is -F_d.  Partials per CTA, three per row.
// ---------------------------------------------------------------------------
constexpr int VT = 256;
__global__ void k_virial_k(DevBox b, const FF *__restrict__ pff,
                           double *part) {
  const FF &ff = *pff;
  int k = blockIdx.x * VT + threadIdx.x;
  double w[3] = {0.0, 0.0, 0.0};
  if (k < b.K) {
    double constVal = 1.0 / (4.0 * ff.alphaSq);
    double factor = b.prefact[k] * (b.sumRref[k] * b.sumRref[k] +
                                    b.sumIref[k] * b.sumIref[k]);
    double c = 2.0 * (constVal + 1.0 / b.hsqr[k]);
    double kv[3] = {b.kx[k], b.ky[k], b.kz[k]};
    for (int d = 0; d < 3; ++d)
      w[d] = factor * (1.0 - c * kv[d] * kv[d]);
  }
  __shared__ double red[VT / 32];
  for (int d = 0; d < 3; ++d) {
    double r = block_sum<VT>(w[d], red);
    if (threadIdx.x == 0)
      part[3 * blockIdx.x + d] = r;
  }
}

__global__ void k_virial_intra(DevBox b, const double *__restrict__ fpart,
                               int nchunk, double *part) {
  int a = blockIdx.x * VT + threadIdx.x;
  double w[3] = {0.0, 0.0, 0.0};
  if (a < b.n_atoms && fabs(b.q[a]) >= 0.000000001) {
    int m = b.mol[a];
    double com[3] = {b.cx[m], b.cy[m], b.cz[m]};
    double pos[3] = {b.x[a], b.y[a], b.z[a]};
    for (int d = 0; d < 3; ++d) {
      double F = 0.0;
      for (int c = 0; c < nchunk; ++c)
        F += fpart[((size_t)c * 3 + d) * b.n_atoms + a];
      double diff = unwrap1(pos[d], com[d], b.L[d], b.half[d]) - com[d];
      w[d] = -F * diff;
    }
  }
  __shared__ double red[VT / 32];
  for (int d = 0; d < 3; ++d) {
    double r = block_sum<VT>(w[d], red);
    if (threadIdx.x == 0)
      part[3 * blockIdx.x + d] = r;
  }
}

__global__ void k_sum3(const double *__restrict__ part, int n, double *out) {
  __shared__ double red[VT / 32];
  for (int d = 0; d < 3; ++d) {
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += VT)
      v += part[3 * i + d];
    double r = block_sum<VT>(v, red);
    if (threadIdx.x == 0)
      out[d] = r;
  }
}

// d_out6: k-space sum (xx, yy, zz), then the intramolecular part
int launch_virial_recip(Box &bx, double *d_out6) {
  DevBox &b = bx.dev;
  int nkb = (b.K + VT - 1) / VT, nab = (b.n_atoms + VT - 1) / VT;
  double *fpart, *kpart;
  int nfp;
  int rc = launch_force_split(bx, b, b.sumRref, b.sumIref,
                              3 * (size_t)(nkb + nab), &fpart, &nfp, &kpart);
  if (rc)
    return rc;
  double *ipart = kpart + 3 * (size_t)nkb;
  k_virial_k<<<nkb, VT, 0, bx.stream>>>(b, bx.d_ff, kpart);
  k_virial_intra<<<nab, VT, 0, bx.stream>>>(b, fpart, nfp, ipart);
  k_sum3<<<1, VT, 0, bx.stream>>>(kpart, nkb, d_out6);
  k_sum3<<<1, VT, 0, bx.stream>>>(ipart, nab, d_out6 + 3);
  return bx.CudaCheck(cudaGetLastError(), "virial recip");
}

}  // namespace gb
