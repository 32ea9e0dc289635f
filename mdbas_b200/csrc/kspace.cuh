// kspace.cuh -- device state of the reciprocal-space sums (ewald_rec.cu,
// spme.cu), shared by the standalone calls and the engine's dynamics.
#pragma once

#include <cufft.h>

#include "common.cuh"

namespace mdbas {

// k-vector list of the explicit Ewald sum for one box / alpha / m-range.
struct EwaldKList {
  bool valid = false;
  double key[12] = {};
  int M1 = 0, M2 = 0, M3 = 0;
  int K = 0, nRows = 0;
  DBuf km, kv, vam, rows, rowK, rowBase, rowPart;
};

struct EwaldWork {
  EwaldKList kl;
  int device = -1;
  DBuf part, S, bpart, sums, tab, pf, done, xyzq, f;
  int parts = 0;      // of the last launch's forces (pf)
  double fact1 = 0.;  // 2 (2 pi / V) C of the last launch
};

// SpmeWork::sums: 0-5 stress, 6 energy, 7-9 force sums
constexpr int kSpmeEnergy = 6, kSpmeForces = 7;
struct SpmeWork {
  int device = -1;
  int m1 = 0, m2 = 0, m3 = 0, nbsp = 0, n = 0;
  cufftHandle plan = 0, planBack = 0;  // D2Z, Z2D
  bool planValid = false, planBackValid = false;
  DBuf qsp, ft, bmod, spl, cell, fr, sums, xyzq, fout;
  // deterministic spreading: atoms binned by the 8^3 grid tile of their
  // base cell, each tile's atoms in ascending index order
  DBuf tileOf, tileCount, tileStart, tileFill, tileList, tileSorted;
  DBuf halo;         // per tile: the (8 + p - 1)^3 halo box of its atoms' stencils
  int haloSmem = 0;  // dynamic shared memory the halo kernel is allowed
  DBuf part;         // per-block partial sums (fixed-order reductions)
  DBuf done;         // their finished-blocks counter
  double f1 = 0.;  // (2 pi / V) C of the last launch
  void drop_plans() {
    if (planValid) cufftDestroy(plan);
    if (planBackValid) cufftDestroy(planBack);
    planValid = planBackValid = false;
  }
  ~SpmeWork() { drop_plans(); }
};

// Explicit Ewald reciprocal forces added to fx/fy/fz (device arrays; with
// scaleInput, MDBas's f = fact0 (f_in + sum) instead of f_in + fact0 sum);
// c.sums[0..6] = {sum_k a_k |S_k|^2, stress sums} on the device.  Once the k
// list and buffers exist for these arguments the call only launches kernels
// (it can be captured into a CUDA graph).
int ewald_launch(EwaldWork &c, int n, const PBC *box, double alpha, double chargeConst, int M1,
                 int M2, int M3, const double *x, const double *y, const double *z,
                 const double *q, double *fx, double *fy, double *fz, int scaleInput,
                 cudaStream_t s);
// SPME reciprocal forces minus their mean added to fx/fy/fz (device arrays);
// c.sums[kSpmeEnergy] = the grid energy sum, c.sums[0..5] stress sums.  Capturable
// once the plan and buffers exist for these arguments.
int spme_launch(SpmeWork &c, int n, const PBC *box, double alpha, double chargeConst, int m1,
                int m2, int m3, int nbsp, const double *x, const double *y, const double *z,
                const double *q, double *fx, double *fy, double *fz, cudaStream_t s);
// Both without the additions when fx is null; these make them.
int ewald_add(EwaldWork &c, int n, double *fx, double *fy, double *fz, int scaleInput,
              cudaStream_t s);
int spme_add(SpmeWork &c, int n, double *fx, double *fy, double *fz, cudaStream_t s);
// sum q and sum q^2 of the self and non-neutral terms.
void charge_sums(int n, const double *q, double *systq, double *sumq2);
// Registers the calls that belong to no engine with host_copy.cuh (once).
void standalone_copies();
// *dst = fixed point (2^-24) of scale * (*src) + add, on the device.
int kspace_fix_launch(const double *src, double scale, double add, long long *dst,
                      cudaStream_t s);

}  // namespace mdbas
