// adjoint.cu -- parameter gradients and force-loss adjoint of the real-space
// Ewald + switched LJ energy (mdbas_nb_engine_adjoint).
//
// The energy is MDBas's (src/energy.c:480-621): per in-cut-off pair of the
// half list E = C q_i q_j erfc(a r)/r + vdw_switch(eps_i eps_j, sig_i + sig_j)
// (src/ewald.c:356-369, src/vdw.c:144-184), per excluded pair
// -C q_i q_j erf(a r)/r (src/ewald.c:371-384), and the self term
// -C a/sqrt(pi) sum q^2 (src/ewald.c:165-171).  For upstream weights v on the
// forces F_i = -dE/dx_i the kernel also returns the gradients of v.F with
// respect to the positions (a Hessian-vector product, -H v) and to the
// per-atom parameters.  With d = x_j - x_i, r = |d|, a pair contributes
// v.F = E'(r) (v_i - v_j).d / r, whose gradient in d is
//   ((v_i - v_j).d / r) (E'' - E'/r) d / r + (E'/r) (v_i - v_j).
// Pair terms are recomputed from the list, never stored.  FP64 throughout:
// the adjoint is the gradient harness's reference-quality path.
#include "common.cuh"
#include "engine.cuh"
#include "host_copy.cuh"
#include "pair_rows.cuh"
#include "real64.cuh"

using namespace mdbas;

namespace {

// Per-unit-charge-product Ewald pair function and its first two radial
// derivatives; `corr` selects the exclusion correction -erf(ar)/r.
struct RadialQ {
  double e, d1, d2;
};

__device__ __forceinline__ RadialQ ewald_unit(const PairParams &p, double r, bool corr) {
  const double ar = p.alpha * r;
  const double g = exp(-(ar * ar));
  const double A = p.chargeConst * 2.0 * p.alpha / kSqrtPi;
  RadialQ o;
  o.e = corr ? -p.chargeConst * erf(ar) / r : p.chargeConst * erfc(ar) / r;
  // E' = -(E + A g)/r holds for both forms, hence E'' = -2E'/r + 2 A a^2 g
  o.d1 = -(o.e + A * g) / r;
  o.d2 = -2.0 * o.d1 / r + 2.0 * A * p.alpha * p.alpha * g;
  return o;
}

// Switched LJ per unit eps_i*eps_j: G, G', G'' and the sigma derivatives
// dG/dsig, dG'/dsig (sig = sig_i + sig_j).
struct RadialLJ {
  double g, d1, d2, s, s1;
};

__device__ __forceinline__ RadialLJ lj_unit(const PairParams &p, double r, double r2,
                                            double sig) {
  RadialLJ o{0., 0., 0., 0., 0.};
  if (!p.vdwSwitch || sig == 0.) return o;
  const double t = sig / r;
  const double s6 = (t * t * t) * (t * t * t);
  const double s12 = s6 * s6;
  const double P = 4.0 * (s12 - s6);
  const double P1 = 24.0 / r * (s6 - 2.0 * s12);
  const double P2 = 4.0 / r2 * (156.0 * s12 - 42.0 * s6);
  const double Ps = 4.0 / sig * (12.0 * s12 - 6.0 * s6);
  const double Ps1 = 24.0 / (r * sig) * (6.0 * s6 - 24.0 * s12);
  if (r2 <= p.cutOn2) {
    o.g = P;
    o.d1 = P1;
    o.d2 = P2;
    o.s = Ps;
    o.s1 = Ps1;
    return o;
  }
  const double a = p.cutOff2 - r2, b = p.cutOn2 - r2;
  const double S = a * a * (p.cutOff2 + 2.0 * r2 - 3.0 * p.cutOn2) * p.switch2;
  const double Su = 6.0 * p.switch2 * a * b;                       // dS/d(r^2)
  const double Suu = -6.0 * p.switch2 * (p.cutOff2 + p.cutOn2 - 2.0 * r2);
  const double S1 = 2.0 * r * Su;
  const double S2 = 2.0 * Su + 4.0 * r2 * Suu;
  o.g = P * S;
  o.d1 = P1 * S + P * S1;
  o.d2 = P2 * S + 2.0 * P1 * S1 + P * S2;
  o.s = Ps * S;
  o.s1 = Ps1 * S + Ps * S1;
  return o;
}

constexpr int kAdjBlocks = 4;  // blocks per SM

struct AdjOut {
  double *gq, *geps, *gsig;   // dE/d(q_i, eps_i, sig_i)
  double *hx, *hy, *hz;       // d(v.F)/dx_i
  double *pq, *peps, *psig;   // d(v.F)/d(q_i, eps_i, sig_i)
};

struct RadialPair {
  RadialQ c;
  RadialLJ l;
};

__device__ __noinline__ RadialPair radial_general(const PairParams &p, double r2, double sig) {
  const double r = sqrt(r2);
  return RadialPair{ewald_unit(p, r, false), lj_unit(p, r, r2, sig)};
}

// The same with the forms of real64.cuh (rt = 1/r, x = alpha r in their
// range, sig an ordinary length or zero).
__device__ __forceinline__ RadialPair radial_fast(const PairParams &p, double r2, double rt,
                                                  double r, double x, double sig) {
  RadialPair o;
  const EwaldConst ek(p);
  const double g = expm64_product(ek.a2, ek.a2lo, r2);
  const double A = p.chargeConst * ek.g0;
  o.c.e = p.chargeConst * (g * erfcx64(x)) * rt;
  o.c.d1 = -(o.c.e + A * g) * rt;
  o.c.d2 = -2.0 * o.c.d1 * rt + 2.0 * A * p.alpha * p.alpha * g;
  o.l = RadialLJ{0., 0., 0., 0., 0.};
  if (!p.vdwSwitch || sig == 0.) return o;
  const double t = sig * rt, t2 = t * t;
  const double s6 = t2 * t2 * t2;
  const double s12 = s6 * s6;
  const double isig = rcp64(sig);
  const double P = 4.0 * (s12 - s6);
  const double P1 = 24.0 * rt * (s6 - 2.0 * s12);
  const double P2 = 4.0 * (rt * rt) * (156.0 * s12 - 42.0 * s6);
  const double Ps = 24.0 * isig * (2.0 * s12 - s6);
  const double Ps1 = 144.0 * (rt * isig) * (s6 - 4.0 * s12);
  const bool inner = r2 <= p.cutOn2;
  const double a = p.cutOff2 - r2, b = p.cutOn2 - r2;
  const double Su = 6.0 * p.switch2 * a * b;
  const double Suu = -6.0 * p.switch2 * (p.cutOff2 + p.cutOn2 - 2.0 * r2);
  const double S =
      inner ? 1. : a * a * (p.cutOff2 + 2.0 * r2 - 3.0 * p.cutOn2) * p.switch2;
  const double S1 = inner ? 0. : 2.0 * r * Su;
  const double S2 = inner ? 0. : 2.0 * Su + 4.0 * r2 * Suu;
  o.l.g = P * S;
  o.l.d1 = P1 * S + P * S1;
  o.l.d2 = P2 * S + 2.0 * P1 * S1 + P * S2;
  o.l.s = Ps * S;
  o.l.s1 = Ps1 * S + Ps * S1;
  return o;
}

// The pairs within the cut-off: the row walk of pair_rows.cuh, j's sums by
// FP64 atomics (9 per pair with force weights, 3 without), i's in registers.
// One thread per atom with the C library's functions took 2.31 ms for 12,000
// atoms (94 blocks, a serial chain of 347 pairs each); this takes 0.32.
template <bool HVP>
__global__ void __launch_bounds__(32 * kRowWarps, kAdjBlocks)
k_adjoint_pairs(int n, DevBox b, PairParams p, HalfList hl, const double *__restrict__ x,
                const double *__restrict__ y, const double *__restrict__ z,
                const double *__restrict__ q, const double *__restrict__ eps,
                const double *__restrict__ sig, int split, const double *__restrict__ vx,
                const double *__restrict__ vy, const double *__restrict__ vz, AdjOut o,
                unsigned *__restrict__ work) {
  __shared__ RowQueue queues[kRowWarps];
  const int lane = threadIdx.x & 31;
  constexpr int N = HVP ? 9 : 3;
  double qi, ei, si, vxi, vyi, vzi, acc[N];
  walk_rows(
      n, split, b, p.cutOff2, hl, x, y, z, queues[threadIdx.x >> 5], work,
      [&](int i) {
        qi = q[i];
        ei = eps[i];
        si = sig[i];
        if constexpr (HVP) {
          vxi = vx[i];
          vyi = vy[i];
          vzi = vz[i];
        }
#pragma unroll
        for (int k = 0; k < N; ++k) acc[k] = 0.;
      },
      [&](int, bool active, int j, double dx, double dy, double dz, double r2) {
        if (!active) return;
        const double qj = q[j], ej = eps[j], sg = si + sig[j];
        const double veps = ei * ej;
        const double rt = rsqrt64(r2), r = sqrt64(r2, rt), xa = p.alpha * r;
        const RadialPair f =
            r2 >= 1e-6 && xa >= 0. && xa <= kErfcxMax && (sg == 0. || (sg >= 1e-3 && sg <= 1e3))
                ? radial_fast(p, r2, rt, r, xa, sg)
                : radial_general(p, r2, sg);
        acc[0] += qj * f.c.e;
        acc[1] += ej * f.l.g;
        acc[2] += veps * f.l.s;
        atomicAdd(o.gq + j, qi * f.c.e);
        atomicAdd(o.geps + j, ei * f.l.g);
        atomicAdd(o.gsig + j, veps * f.l.s);
        if constexpr (HVP) {
          const double ux = vxi - vx[j], uy = vyi - vy[j], uz = vzi - vz[j];
          const double ud = (ux * dx + uy * dy + uz * dz) * rt;  // (v_i - v_j).d / r
          const double qq = qi * qj;
          const double E1 = qq * f.c.d1 + veps * f.l.d1;
          const double E2 = qq * f.c.d2 + veps * f.l.d2;
          const double bb = E1 * rt, a = ud * (E2 - bb) * rt;
          const double hx = a * dx + bb * ux, hy = a * dy + bb * uy, hz = a * dz + bb * uz;
          acc[3] -= hx;
          acc[4] -= hy;
          acc[5] -= hz;
          atomicAdd(o.hx + j, hx);
          atomicAdd(o.hy + j, hy);
          atomicAdd(o.hz + j, hz);
          const double cd = f.c.d1 * ud, ld = f.l.d1 * ud, ls = veps * f.l.s1 * ud;
          acc[6] += qj * cd;
          acc[7] += ej * ld;
          acc[8] += ls;
          atomicAdd(o.pq + j, qi * cd);
          atomicAdd(o.peps + j, ei * ld);
          atomicAdd(o.psig + j, ls);
        }
      },
      [&](int i) {
        double *const dst[9] = {o.gq, o.geps, o.gsig, o.hx, o.hy, o.hz, o.pq, o.peps, o.psig};
#pragma unroll
        for (int k = 0; k < N; ++k) {
          const double v = warp_sum_d(acc[k]);
          if (lane == 0) atomicAdd(dst[k] + i, v);
        }
      });
}

// An excluded pair's terms into acc (atom i) and by atomics (atom j).
__device__ __forceinline__ void adj_excluded(const PairParams &p, int i, int j, double dx,
                                             double dy, double dz, double r2, const double *q,
                                             const double *vx, const double *vy,
                                             const double *vz, const AdjOut &o,
                                             double (&acc)[5]) {
  const double r = sqrt(r2);
  const double qi = q[i], qj = q[j];
  const RadialQ c = ewald_unit(p, r, true);
  acc[0] += qj * c.e;
  atomicAdd(o.gq + j, qi * c.e);
  if (!vx) return;
  const double ux = vx[i] - vx[j], uy = vy[i] - vy[j], uz = vz[i] - vz[j];
  const double ud = (ux * dx + uy * dy + uz * dz) / r;
  const double E1 = qi * qj * c.d1, E2 = qi * qj * c.d2;
  const double a = ud * (E2 - E1 / r) / r, b = E1 / r;
  const double hx = a * dx + b * ux, hy = a * dy + b * uy, hz = a * dz + b * uz;
  acc[1] -= hx;
  acc[2] -= hy;
  acc[3] -= hz;
  atomicAdd(o.hx + j, hx);
  atomicAdd(o.hy + j, hy);
  atomicAdd(o.hz + j, hz);
  acc[4] += qj * c.d1 * ud;
  atomicAdd(o.pq + j, qi * c.d1 * ud);
}

// Excluded pairs (j > i of each row, no cut-off) and the self term.
__global__ void __launch_bounds__(128)
k_adjoint_excl(int n, DevBox b, PairParams p, const int *__restrict__ exclStart,
               const int *__restrict__ exclFlat, const double *__restrict__ x,
               const double *__restrict__ y, const double *__restrict__ z,
               const double *__restrict__ q, const double *__restrict__ vx,
               const double *__restrict__ vy, const double *__restrict__ vz, AdjOut o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double acc[5] = {0., 0., 0., 0., 0.};
  acc[0] = -2.0 * p.chargeConst * p.alpha * q[i] / kSqrtPi;  // self term
  const int e = exclStart[i + 1];
  for (int k = exclStart[i]; k < e; ++k) {
    const int j = exclFlat[k];
    if (j <= i) continue;
    double dx = x[j] - x[i], dy = y[j] - y[i], dz = z[j] - z[i];
    const double r2 = dist_d(b, dx, dy, dz);
    adj_excluded(p, i, j, dx, dy, dz, r2, q, vx, vy, vz, o, acc);
  }
  atomicAdd(o.gq + i, acc[0]);
  if (!vx) return;
  atomicAdd(o.hx + i, acc[1]);
  atomicAdd(o.hy + i, acc[2]);
  atomicAdd(o.hz + i, acc[3]);
  atomicAdd(o.pq + i, acc[4]);
}

}  // namespace

extern "C" int mdbas_nb_engine_adjoint(mdbas_nb_engine *e, const double *vx, const double *vy,
                                       const double *vz, double *gq, double *geps, double *gsig,
                                       double *hx, double *hy, double *hz, double *pq,
                                       double *peps, double *psig, int device_ptrs) {
  if (!e || !gq || !geps || !gsig) return MDBAS_NB_ERR_ARG;
  const bool hvp = vx != nullptr;
  if (hvp && (!vy || !vz || !hx || !hy || !hz || !pq || !peps || !psig)) return MDBAS_NB_ERR_ARG;
  if (e->cfg.precision != 0) {
    set_last_status(MDBAS_NB_ERR_UNSUPPORTED, "the adjoint runs on the FP64 form (precision 0)");
    return MDBAS_NB_ERR_UNSUPPORTED;
  }
  if (!e->built) return MDBAS_NB_ERR_STATE;
  MDB_CUDA(cudaSetDevice(e->device));
  LaunchScope ls(e);
  const int n = e->n;
  cudaStream_t s = e->stream;
  // device scratch: 3 (v) + 9 (outputs) arrays of n and the work counter
  MDB_TRY(e->adjBuf.ensure(sizeof(double) * (12 * (size_t)n + 1)));
  double *buf = e->adjBuf.as<double>();
  double *dv = buf, *outs = buf + 3 * (size_t)n;
  MDB_CUDA(cudaMemsetAsync(outs, 0, sizeof(double) * (9 * (size_t)n + 1), s));
  const size_t bytes = sizeof(double) * (size_t)n;
  if (hvp && device_ptrs) {
    const cudaMemcpyKind k = cudaMemcpyDeviceToDevice;
    MDB_CUDA(cudaMemcpyAsync(dv, vx, bytes, k, s));
    MDB_CUDA(cudaMemcpyAsync(dv + n, vy, bytes, k, s));
    MDB_CUDA(cudaMemcpyAsync(dv + 2 * (size_t)n, vz, bytes, k, s));
  } else if (hvp) {
    const CopySpan3 in(const_cast<double *>(vx), const_cast<double *>(vy),
                       const_cast<double *>(vz), dv, n);
    MDB_TRY(copy_in(in.s, 3, s));
  }
  AdjOut o;
  double *const ptrs[9] = {outs, outs + n, outs + 2 * (size_t)n, outs + 3 * (size_t)n,
                           outs + 4 * (size_t)n, outs + 5 * (size_t)n, outs + 6 * (size_t)n,
                           outs + 7 * (size_t)n, outs + 8 * (size_t)n};
  o.gq = ptrs[0]; o.geps = ptrs[1]; o.gsig = ptrs[2];
  o.hx = ptrs[3]; o.hy = ptrs[4]; o.hz = ptrs[5];
  o.pq = ptrs[6]; o.peps = ptrs[7]; o.psig = ptrs[8];
  const double *dvx = hvp ? dv : nullptr, *dvy = hvp ? dv + n : nullptr,
               *dvz = hvp ? dv + 2 * (size_t)n : nullptr;
  const RowGrid g = row_grid(n, kAdjBlocks);
  const HalfList hl{e->ref.order.as<int>(), e->ref.neighPair.as<int>(),
                    e->ref.off.as<long long>(), e->ref.list.as<int>()};
  const auto kern = hvp ? k_adjoint_pairs<true> : k_adjoint_pairs<false>;
  MDB_LAUNCH(kern, g.blocks, 32 * kRowWarps, 0, s, n, e->box, e->pp, hl, e->x.as<double>(),
             e->y.as<double>(), e->z.as<double>(), e->q.as<double>(), e->eps.as<double>(),
             e->sig.as<double>(), g.split, dvx, dvy, dvz, o,
             reinterpret_cast<unsigned *>(outs + 9 * (size_t)n));
  MDB_LAUNCH(k_adjoint_excl, grid_for(n, 128), 128, 0, s, n, e->box, e->pp,
             e->exclStart.as<int>(), e->exclFlat.as<int>(), e->x.as<double>(),
             e->y.as<double>(), e->z.as<double>(), e->q.as<double>(), dvx, dvy, dvz, o);
  double *dst[9] = {gq, geps, gsig, hx, hy, hz, pq, peps, psig};
  const int outputs = hvp ? 9 : 3;
  if (!device_ptrs) {
    CopySpan out[9];
    for (int k = 0; k < outputs; ++k) out[k] = CopySpan(dst[k], ptrs[k], bytes, false, k > 0);
    return copy_out(out, outputs, s);
  }
  for (int k = 0; k < outputs; ++k)
    MDB_CUDA(cudaMemcpyAsync(dst[k], ptrs[k], bytes, cudaMemcpyDeviceToDevice, s));
  MDB_CUDA(cudaStreamSynchronize(s));
  return MDBAS_NB_OK;
}
