// pair_fp64.cu -- the plain FP64 GPU form of MDBas's pair loops.
//
// One warp per atom i (in neighOrder position), over i's entries of the
// MDBas half list as ewald_energy / nonbond_energy take them
// (src/energy.c:480-561, :240-318): min-image by dist(), cut-off test,
// Ewald direct (src/ewald.c:356-369) or cut-off Coulomb (src/elec.c:137-263)
// plus vdw_switch (src/vdw.c:144-184), Newton's third law with the j update
// done by an FP64 atomic.  Exclusion corrections (src/energy.c:567-621) run
// one thread per atom over its j>i exclusion rows.
//
// This translation unit is compiled with --fmad=false.  Distances, the cut-off
// test and the general pair form keep MDBas's association order; the Ewald
// pairs of the ordinary range take the Newton and polynomial forms of
// real64.cuh (a few ulp from the C library's; no further from exact).  The
// order of the FP64 additions is not fixed.
#include "common.cuh"
#include "pair_fp64.cuh"
#include "pair_rows.cuh"
#include "real64.cuh"

namespace mdbas {

namespace {

__device__ __forceinline__ double ewald_dir_d(const PairParams &p, double &dE, double qel, double r,
                                              double rt) {
  const double alphar = p.alpha * r;
  const double e = qel * erfc(alphar) * rt;
  dE = 2.0 * qel * p.alpha * exp(-(alphar * alphar)) / kSqrtPi;
  dE = -(e + dE) * rt;
  return e;
}

__device__ __forceinline__ double ewald_corr_d(const PairParams &p, double &dE, double qel,
                                               double r, double rt) {
  const double alphar = p.alpha * r;
  const double e = -qel * erf(alphar) * rt;
  dE = 2.0 * qel * p.alpha * exp(-(alphar * alphar)) / kSqrtPi;
  dE = -(e + dE) * rt;
  return e;
}

__device__ __forceinline__ double vdw_switch_d(const PairParams &p, double &dvdw, double veps,
                                               double vsig, double r2, double rt) {
  if (!p.vdwSwitch) {
    dvdw = 0.;
    return 0.;
  }
  const double t = vsig * rt;
  const double v6 = (t * t * t) * (t * t * t);
  const double v12 = v6 * v6;
  if (r2 <= p.cutOn2) {
    dvdw = 24. * veps * rt * (v6 - 2. * v12);
    return 4. * veps * (v12 - v6);
  }
  const double s1 = p.cutOff2 - r2;
  const double sf = (s1 * s1) * (p.cutOff2 + 2. * r2 - 3. * p.cutOn2) * p.switch2;
  const double dsf = 12. * r2 * s1 * (p.cutOn2 - r2) * p.switch2;
  const double pv = 4. * veps * (v12 - v6);
  const double dpv = 24. * veps * (v6 - 2. * v12);
  dvdw = pv * dsf + dpv * sf;
  dvdw *= rt;
  return pv * sf;
}

// coulomb_shift1 / shift2 / switch / none (src/elec.c:25-263).
__device__ __forceinline__ double coulomb_d(const PairParams &p, double &delec, double qel,
                                            double r2, double rt) {
  double s1, s2, sf, dsf, pelec;
  switch (p.elecType) {
    case SHIFT1:
      s1 = rt * r2 * p.rcutOff;
      s2 = r2 * p.rcutOff2;
      sf = 1. - 2. * s1 + s2;
      dsf = 2. * (s2 - s1);
      pelec = p.chargeConst * qel * rt;
      delec = pelec * rt * (dsf - sf);
      return pelec * sf;
    case SHIFT2:
      s1 = r2 * p.rcutOff2;
      s2 = s1 * s1;
      sf = 1. - 2. * s1 + s2;
      dsf = 4. * (s2 - s1);
      pelec = p.chargeConst * qel * rt;
      delec = pelec * rt * (dsf - sf);
      return pelec * sf;
    case SWITCH:
      if (r2 <= p.cutOn2) {
        pelec = p.chargeConst * qel * rt;
        delec = -pelec * rt;
        return pelec;
      }
      s1 = p.cutOff2 - r2;
      sf = (s1 * s1) * (p.cutOff2 + 2. * r2 - 3. * p.cutOn2) * p.switch2;
      dsf = 12. * r2 * s1 * (p.cutOn2 - r2) * p.switch2;
      pelec = p.chargeConst * qel * rt;
      delec = pelec * rt * (dsf - sf);
      return pelec * sf;
    default:
      delec = 0.;
      return 0.;
  }
}

// One in-cut-off pair: energies, r dE/dr of each term and the force factor
// f = (dE/dr) / r.
struct PairTerms {
  double eel, evdw, wel, wvdw, f;
};

// MDBas's expressions with the C library's sqrt, erfc and exp: the cut-off
// Coulomb forms, and the Ewald pairs that pair_ewald_fast does not take.
template <bool EWALD>
__device__ __forceinline__ PairTerms pair_general(const PairParams &p, double qq, double veps,
                                                  double vsig, double r2) {
  PairTerms o;
  double delec, dvdw;
  const double r = sqrt(r2);
  const double rt = 1. / r;
  if (EWALD)
    o.eel = ewald_dir_d(p, delec, qq, r, rt);
  else
    o.eel = coulomb_d(p, delec, qq, r2, rt);
  o.evdw = vdw_switch_d(p, dvdw, veps, vsig, r2, rt);
  o.wel = delec * r;
  o.wvdw = dvdw * r;
  o.f = (delec + dvdw) * rt;
  return o;
}

__device__ __noinline__ PairTerms pair_ewald_slow(const PairParams &p, double qq, double veps,
                                                  double vsig, double r2) {
  return pair_general<true>(p, qq, veps, vsig, r2);
}

// The same Ewald pair with the forms of real64.cuh; the caller has checked
// that r2 and alpha r lie in their range.
__device__ __forceinline__ PairTerms pair_ewald_fast(const PairParams &p, const EwaldConst &k,
                                                     double qq, double veps, double vsig,
                                                     double r2, double rt, double x) {
  PairTerms o;
  const double g = expm64_product(k.a2, k.a2lo, r2);
  o.eel = qq * (g * erfcx64(x)) * rt;
  o.wel = -fma(k.g0 * qq, g, o.eel);
  o.evdw = o.wvdw = 0.;
  if (p.vdwSwitch) {
    const double t = vsig * rt;
    const double t2 = t * t;
    const double v6 = t2 * t2 * t2;
    const double ve4 = 4. * veps;
    const double pv = ve4 * fma(v6, v6, -v6);
    const double dpv = 6. * ve4 * fma(-2. * v6, v6, v6);
    const double s1 = p.cutOff2 - r2, s2 = s1 * k.sw2;
    const bool inner = r2 <= p.cutOn2;
    const double sf = inner ? 1. : s1 * s2 * fma(2., r2, k.swc);
    const double dsf = inner ? 0. : 12. * r2 * s2 * (p.cutOn2 - r2);
    o.evdw = pv * sf;
    o.wvdw = fma(pv, dsf, dpv * sf);
  }
  const double r2inv = rt * rt;
  o.f = (o.wel + o.wvdw) * fma(fma(-r2, r2inv, 1.0), r2inv, r2inv);
  return o;
}

// Smallest r2 of the fast form: far below any atomic distance, far above
// where its powers of 1/r could overflow.
constexpr double kFastR2Min = 1e-6;
constexpr int kPairBlocks = 6;    // blocks per SM

// The sum of every block's v into acc[c], without the rounding of one FP64
// addition after the other (a thousand blocks' would show in differences of
// energies): multiples of 2^-10 and what is left of v, in multiples of 2^-60,
// are added as integers, and the last block puts them together.  What v holds
// below 2^-60 (nothing from 2^-7 on; all of a weak pair's energy of 1e-19) and
// sums too large for the integers are added as they are.
__device__ __forceinline__ void exact_add(double *acc, int c, double v) {
  if (!(fabs(v) < 1e12)) {
    atomicAdd(acc + c, v);
    return;
  }
  const long long h = __double2ll_rn(v * 1024.);
  double rest = v - (double)h * (1. / 1024.);
  const long long l = __double2ll_rn(rest * 1152921504606846976.);
  rest -= (double)l * (1. / 1152921504606846976.);
  red_add(reinterpret_cast<long long *>(acc + 8 + 2 * c), h);
  red_add(reinterpret_cast<long long *>(acc + 9 + 2 * c), l);
  if (rest != 0.) atomicAdd(acc + c, rest);
}
__device__ __forceinline__ void exact_finish(double *acc, int c) {
  const long long h = __ldcg(reinterpret_cast<long long *>(acc + 8 + 2 * c));
  const long long l = __ldcg(reinterpret_cast<long long *>(acc + 9 + 2 * c));
  atomicAdd(acc + c, (double)h * (1. / 1024.) + (double)l * (1. / 1152921504606846976.));
}

// acc: see pair_fp64.cuh.
//
// The row walk of pair_rows.cuh; warps keep their energy sums in registers
// over all their atoms.  Bound by latency and the LSU (gathers and scattered
// additions, 60% of the data-pipe cycles; FP64 pipe 40%).  Measured against
// one thread per atom with the C library's functions: 2.26 -> 0.67 ms at
// 96,000 atoms of water, 1.22 -> 0.10 at 12,000, 1.23 -> 0.046 at 3,000 (calls
// in a row, L2 warm; 0.79 at 96,000 after an L2 flush).  Atoms packed to one 32-byte sector and j forces added a sector at a time
// measured no better (0.67 and 1.1 ms).
template <bool EWALD>
__global__ void __launch_bounds__(32 * kRowWarps, kPairBlocks)
k_pairs_fp64(int n, DevBox b, PairParams p, HalfList hl, const double *__restrict__ x,
             const double *__restrict__ y, const double *__restrict__ z,
             const double *__restrict__ q, const double *__restrict__ eps,
             const double *__restrict__ sig, int split, double *__restrict__ fx,
             double *__restrict__ fy, double *__restrict__ fz, double *__restrict__ acc) {
  __shared__ RowQueue queues[kRowWarps];
  __shared__ double red[5][kRowWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const EwaldConst ek(p);
  double eel = 0., evdw = 0., virel = 0., virvdw = 0.;
  int npair = 0;
  double qi, ei, si, fxi, fyi, fzi;
  walk_rows(
      n, split, b, p.cutOff2, hl, x, y, z, queues[w], reinterpret_cast<unsigned *>(acc + 7),
      [&](int i) {
        qi = EWALD ? p.chargeConst * q[i] : q[i];
        ei = eps[i];
        si = sig[i];
        fxi = fyi = fzi = 0.;
      },
      [&](int take, bool active, int j, double dx, double dy, double dz, double r2) {
        npair += take;
        if (!active) return;
        const double qq = qi * q[j], veps = ei * eps[j], vsig = si + sig[j];
        PairTerms o;
        if constexpr (EWALD) {
          const double rt = rsqrt64(r2);
          const double xa = p.alpha * sqrt64(r2, rt);
          if (r2 >= kFastR2Min && xa >= 0. && xa <= kErfcxMax)
            o = pair_ewald_fast(p, ek, qq, veps, vsig, r2, rt, xa);
          else
            o = pair_ewald_slow(p, qq, veps, vsig, r2);
        } else {
          o = pair_general<false>(p, qq, veps, vsig, r2);
        }
        eel += o.eel;
        evdw += o.evdw;
        virel += o.wel;
        virvdw += o.wvdw;
        const double fxj = o.f * dx, fyj = o.f * dy, fzj = o.f * dz;
        fxi += fxj;
        fyi += fyj;
        fzi += fzj;
        atomicAdd(fx + j, -fxj);
        atomicAdd(fy + j, -fyj);
        atomicAdd(fz + j, -fzj);
      },
      [&](int i) {
        fxi = warp_sum_d(fxi);
        fyi = warp_sum_d(fyi);
        fzi = warp_sum_d(fzi);
        if (lane < 3) {
          const double v = lane == 0 ? fxi : lane == 1 ? fyi : fzi;
          atomicAdd((lane == 0 ? fx : lane == 1 ? fy : fz) + i, v);
        }
      });
  const double sum[4] = {warp_sum_d(eel), warp_sum_d(evdw), warp_sum_d(virel),
                         warp_sum_d(virvdw)};
  if (lane == 0) {
    for (int c = 0; c < 4; ++c) red[c][w] = sum[c];
    red[4][w] = (double)npair;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    double v = 0.;
    for (int c = 0; c < kRowWarps; ++c) v += red[threadIdx.x][c];
    exact_add(acc, threadIdx.x, v);
    __threadfence();
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicAdd(reinterpret_cast<unsigned *>(acc + 7) + 1, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last && threadIdx.x < 5) {
    __threadfence();
    exact_finish(acc, threadIdx.x);
  }
}

// Exclusion correction (src/energy.c:567-621): every excluded pair j>i, no
// cut-off.  acc[5], acc[6]: eCorr, virCorr.
__global__ void __launch_bounds__(128)
k_excl_fp64(int n, DevBox b, PairParams p, const int *__restrict__ exclStart,
            const int *__restrict__ exclFlat, const double *__restrict__ x,
            const double *__restrict__ y, const double *__restrict__ z,
            const double *__restrict__ q, double *__restrict__ fx, double *__restrict__ fy,
            double *__restrict__ fz, double *__restrict__ acc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ecorr = 0., vcorr = 0.;
  if (i < n) {
    double fxi = 0., fyi = 0., fzi = 0.;
    const int e = exclStart[i + 1];
    for (int k = exclStart[i]; k < e; ++k) {
      const int j = exclFlat[k];
      if (j <= i) continue;
      double dx = x[j] - x[i], dy = y[j] - y[i], dz = z[j] - z[i];
      const double r2 = dist_d(b, dx, dy, dz);
      const double r = sqrt(r2);
      const double rt = 1. / r;
      const double qel = p.chargeConst * q[i] * q[j];
      double dE;
      ecorr += ewald_corr_d(p, dE, qel, r, rt);
      vcorr += dE * r;
      const double fxj = dE * dx * rt;
      const double fyj = dE * dy * rt;
      const double fzj = dE * dz * rt;
      fxi += fxj;
      fyi += fyj;
      fzi += fzj;
      atomicAdd(fx + j, -fxj);
      atomicAdd(fy + j, -fyj);
      atomicAdd(fz + j, -fzj);
    }
    if (fxi != 0. || fyi != 0. || fzi != 0.) {
      atomicAdd(fx + i, fxi);
      atomicAdd(fy + i, fyi);
      atomicAdd(fz + i, fzi);
    }
  }
  ecorr = warp_sum_d(ecorr);
  vcorr = warp_sum_d(vcorr);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(acc + 5, ecorr);
    atomicAdd(acc + 6, vcorr);
  }
}

// Ewald self term (src/ewald.c:165-171): sum q^2, each term rounded to a
// multiple of 2^-40 and summed as an integer, so the total does not depend on
// the atom order.  *acc receives the int64 sum.
__global__ void k_sum_q2(int n, const double *__restrict__ q, long long *__restrict__ acc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  long long v = (i < n) ? __double2ll_rn(q[i] * q[i] * 1099511627776.0) : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red_add(acc, v);
}

// 1-4 pairs: ewald14_energy (src/energy.c:654-742) with ewald_dir14/corr14
// (src/ewald.c:386-413) and vdw14_switch (src/vdw.c:270-311), or
// nonbond14_energy (src/energy.c:356-439) with coulomb14_* (src/elec.c:265-465).
// One thread per pair; acc[0..3] += elec, vdw, virelec, virvdw.
template <bool EWALD>
__global__ void __launch_bounds__(128)
k_pairs14(int npair, DevBox b, PairParams p, const int *__restrict__ list14,
          const double *__restrict__ x, const double *__restrict__ y,
          const double *__restrict__ z, const double *__restrict__ q,
          const double *__restrict__ eps, const double *__restrict__ sig,
          double *__restrict__ fx, double *__restrict__ fy, double *__restrict__ fz,
          double *__restrict__ acc) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double eel = 0., evdw = 0., virel = 0., virvdw = 0.;
  if (k < npair) {
    const int i = list14[2 * k], j = list14[2 * k + 1];
    double dx = x[j] - x[i], dy = y[j] - y[i], dz = z[j] - z[i];
    const double r2 = dist_d(b, dx, dy, dz);
    const double r = sqrt(r2);
    const double rt = 1. / r;
    double delec = 0., dcorr = 0., dvdw = 0.;
    if (EWALD) {
      const double qel = p.chargeConst * q[i] * q[j];
      const double alphar = p.alpha * r;
      const double ed = p.scal14 * qel * erfc(alphar) * rt;
      delec = 2.0 * p.scal14 * qel * p.alpha * exp(-(alphar * alphar)) / kSqrtPi;
      delec = -(ed + delec) * rt;
      const double ec = (p.scal14 - 1.0) * qel * erf(alphar) * rt;
      dcorr = 2.0 * (p.scal14 - 1.0) * qel * p.alpha * exp(-(alphar * alphar)) / kSqrtPi;
      dcorr = (dcorr - ec) * rt;
      eel = ed + ec;
      virel = delec * r + dcorr * r;
    } else {
      const double qel = q[i] * q[j];
      double s1, s2, sf, dsf, pelec;
      switch (p.elecType) {
        case SHIFT1:
          if (r2 <= p.cutOff2) {
            s1 = rt * r2 * p.rcutOff;
            s2 = r2 * p.rcutOff2;
            sf = 1. - 2. * s1 + s2;
            dsf = 2. * (s2 - s1);
            pelec = p.scal14 * p.chargeConst * qel * rt;
            eel = pelec * sf;
            delec = pelec * rt * (dsf - sf);
          }
          break;
        case SHIFT2:
          if (r2 <= p.cutOff2) {
            s1 = r2 * p.rcutOff2;
            s2 = s1 * s1;
            sf = 1. - 2. * s1 + s2;
            dsf = 4. * (s2 - s1);
            pelec = p.scal14 * p.chargeConst * qel * rt;
            eel = pelec * sf;
            delec = pelec * rt * (dsf - sf);
          }
          break;
        case SWITCH:
          if (r2 <= p.cutOn2) {
            pelec = p.scal14 * p.chargeConst * qel * rt;
            eel = pelec;
            delec = -pelec * rt;
          } else if (r2 <= p.cutOff2) {
            s1 = p.cutOff2 - r2;
            sf = (s1 * s1) * (p.cutOff2 + 2. * r2 - 3. * p.cutOn2) * p.switch2;
            dsf = 12. * r2 * s1 * (p.cutOn2 - r2) * p.switch2;
            pelec = p.scal14 * p.chargeConst * qel * rt;
            eel = pelec * sf;
            delec = pelec * rt * (dsf - sf);
          }
          break;
        default:
          break;
      }
      virel = delec * r;
    }
    if (p.vdwSwitch) {
      const double veps = eps[i] * eps[j], vsig = sig[i] + sig[j];
      const double t = vsig * rt;
      const double v6 = (t * t * t) * (t * t * t);
      const double v12 = v6 * v6;
      if (r2 <= p.cutOn2) {
        evdw = 4. * p.scal14 * veps * (v12 - v6);
        dvdw = 24. * p.scal14 * veps * rt * (v6 - 2. * v12);
      } else if (r2 <= p.cutOff2) {
        const double s1 = p.cutOff2 - r2;
        const double sf = (s1 * s1) * (p.cutOff2 + 2. * r2 - 3. * p.cutOn2) * p.switch2;
        const double dsf = 12. * r2 * s1 * (p.cutOn2 - r2) * p.switch2;
        const double pv = 4. * p.scal14 * veps * (v12 - v6);
        const double dpv = 24. * p.scal14 * veps * (v6 - 2. * v12);
        evdw = pv * sf;
        dvdw = pv * dsf + dpv * sf;
        dvdw *= rt;
      }
    }
    virvdw = dvdw * r;
    const double fxj = (delec + dcorr + dvdw) * dx * rt;
    const double fyj = (delec + dcorr + dvdw) * dy * rt;
    const double fzj = (delec + dcorr + dvdw) * dz * rt;
    atomicAdd(fx + i, fxj);
    atomicAdd(fy + i, fyj);
    atomicAdd(fz + i, fzj);
    atomicAdd(fx + j, -fxj);
    atomicAdd(fy + j, -fyj);
    atomicAdd(fz + j, -fzj);
  }
  eel = warp_sum_d(eel);
  evdw = warp_sum_d(evdw);
  virel = warp_sum_d(virel);
  virvdw = warp_sum_d(virvdw);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(acc + 0, eel);
    atomicAdd(acc + 1, evdw);
    atomicAdd(acc + 2, virel);
    atomicAdd(acc + 3, virvdw);
  }
}

}  // namespace

int pairs_fp64(int ewald, int n, const DevBox &b, const PairParams &p, const int *order,
               const int *neighPair, const long long *off, const int *list, const double *x,
               const double *y, const double *z, const double *q, const double *eps,
               const double *sig, double *fx, double *fy, double *fz, double *acc,
               cudaStream_t s) {
  if (n <= 0) return MDBAS_NB_OK;
  const RowGrid g = row_grid(n, kPairBlocks);
  const HalfList hl{order, neighPair, off, list};
  const auto kern = ewald ? k_pairs_fp64<true> : k_pairs_fp64<false>;
  MDB_LAUNCH(kern, g.blocks, 32 * kRowWarps, 0, s, n, b, p, hl, x, y, z, q, eps, sig, g.split, fx,
             fy, fz, acc);
  return MDBAS_NB_OK;
}

int excl_fp64(int n, const DevBox &b, const PairParams &p, const int *exclStart,
              const int *exclFlat, const double *x, const double *y, const double *z,
              const double *q, double *fx, double *fy, double *fz, double *acc,
              cudaStream_t s) {
  if (n <= 0) return MDBAS_NB_OK;
  MDB_LAUNCH(k_excl_fp64, grid_for(n, 128), 128, 0, s, n, b, p, exclStart, exclFlat, x, y, z, q,
             fx, fy, fz, acc);
  return MDBAS_NB_OK;
}

int pairs14_fp64(int ewald, int npair, const DevBox &b, const PairParams &p, const int *list14,
                 const double *x, const double *y, const double *z, const double *q,
                 const double *eps, const double *sig, double *fx, double *fy, double *fz,
                 double *acc, cudaStream_t s) {
  if (npair <= 0) return MDBAS_NB_OK;
  if (ewald)
    MDB_LAUNCH(k_pairs14<true>, grid_for(npair, 128), 128, 0, s, npair, b, p, list14, x, y, z, q,
               eps, sig, fx, fy, fz, acc);
  else
    MDB_LAUNCH(k_pairs14<false>, grid_for(npair, 128), 128, 0, s, npair, b, p, list14, x, y, z,
               q, eps, sig, fx, fy, fz, acc);
  return MDBAS_NB_OK;
}

int sum_q2(int n, const double *q, long long *acc, cudaStream_t s) {
  if (n <= 0) return MDBAS_NB_OK;
  MDB_LAUNCH(k_sum_q2, grid_for(n, 256), 256, 0, s, n, q, acc);
  return MDBAS_NB_OK;
}

}  // namespace mdbas
