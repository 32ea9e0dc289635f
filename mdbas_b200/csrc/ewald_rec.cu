// ewald_rec.cu -- MDBas's explicit reciprocal-space Ewald sum on the GPU:
// init_ewald, ewald_free and ewald_rec (include/ewald.h; src/ewald.c:10-354).
//
// MDBas sums over every k = 2 pi (m1 u + m2 v + m3 w) inside the reciprocal
// cut-off, in the order m1 = 0..m1max, m2, m3 (half space: the (0, 0, m3 > 0)
// row first), with per-atom tables of cos/sin(m s) built by the angle-
// addition recurrence.  Here:
//
//   * the k list (and e^{-k^2/4a^2}/k^2, the virial factor) is built on the
//     host with MDBas's expressions and cached per box, alpha and m-range;
//   * k_ewald_tables: the atoms' cos/sin tables, by MDBas's recurrence, once;
//   * k_ewald_sf: one thread per k-vector sums q_i e^{i k.r_i} over a range
//     of atoms, a tile of their tables at a time in shared memory; partial
//     sums per atom range are added in a fixed order by k_ewald_kdata
//     (deterministic);
//   * k_ewald_forces: one thread per atom and part of the k list (rows of
//     fixed (m1, m2), m3 contiguous); a row's terms share the vector of its
//     first two indices, so per k only the two sums over m3 are needed;
//   * k_ewald_add: the parts added in order, scaled, into the forces.
//
// This file is compiled with --fmad=false (the table recurrences are MDBas's
// operations); products and sums over k and atoms use FMAs and an order of
// their own.
#include <math.h>
#include <string.h>

#include <vector>

#include "host_copy.cuh"
#include "kspace.cuh"

namespace mdbas {
namespace {

constexpr double kTwoPi = 6.283185307179586;  // include/global.h:54
constexpr double kPi = 3.141592653589793;
constexpr int kSfThreads = 256;               // k-vectors per structure-factor block
constexpr int kEwParts = 32;                  // most parts of the force kernel's k list

struct EwBox {
  double u1, u2, u3, v1, v2, v3, w1, w2, w3;
};

// scaled fractional coordinate of one dimension, MDBas's expression
__device__ __forceinline__ double frac_s(const EwBox &b, int d, double x, double y, double z) {
  if (d == 0) return kTwoPi * (x * b.u1 + y * b.u2 + z * b.u3);
  if (d == 1) return kTwoPi * (x * b.v1 + y * b.v2 + z * b.v3);
  return kTwoPi * (x * b.w1 + y * b.w2 + z * b.w3);
}

// c[m] = cos(m s), sn[m] = sin(m s) for m = 0..M by MDBas's recurrence
// (src/ewald.c:196-227); stride between entries `st`.
__device__ __forceinline__ void ew_table(double s, int M, double *c, double *sn, int st) {
  c[0] = 1.0;
  sn[0] = 0.0;
  if (M < 1) return;
  const double c1 = cos(s), s1 = sin(s);
  c[st] = c1;
  sn[st] = s1;
  double cp = c1, sp = s1;
  for (int m = 2; m <= M; ++m) {
    const double cn = cp * c1 - sp * s1;
    const double snn = sp * c1 + cp * s1;
    c[(size_t)m * st] = cn;
    sn[(size_t)m * st] = snn;
    cp = cn;
    sp = snn;
  }
}

// The tables of all atoms, entry e of atom i at tab[e n + i]; entries in the
// order cos(m s1), sin(m s1), m = 0..M1, then dimension 2 and 3.  One thread
// per atom and dimension (grid y).
__global__ void __launch_bounds__(128)
    k_ewald_tables(int n, EwBox b, int M1, int M2, int M3, const double *__restrict__ x,
                   const double *__restrict__ y, const double *__restrict__ z,
                   double *__restrict__ tab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int d = blockIdx.y;
  const int M = d == 0 ? M1 : d == 1 ? M2 : M3;
  const int e = d == 0 ? 0 : d == 1 ? 2 * (M1 + 1) : 2 * (M1 + M2 + 2);
  double *c = tab + (size_t)e * n + i;
  ew_table(frac_s(b, d, x[i], y[i], z[i]), M, c, c + (size_t)(M + 1) * n, n);
}

// Structure factors: part[(2p) K + k], part[(2p+1) K + k] = sum over the atoms
// of range p of q_i cos(k.r_i), q_i sin(k.r_i).
__global__ void __launch_bounds__(kSfThreads)
    k_ewald_sf(int n, int K, int perPart, int tile, int M1, int M2, int M3,
               const int4 *__restrict__ km, const double *__restrict__ tab,
               const double *__restrict__ q, double *__restrict__ part) {
  extern __shared__ double sh[];
  const int W = 2 * (M1 + M2 + M3 + 3);  // doubles per atom
  const int st = W | 1;                  // odd stride: no bank conflicts on the way in
  const int o1s = M1 + 1, o2c = 2 * (M1 + 1), o2s = o2c + M2 + 1, o3c = o2s + M2 + 1,
            o3s = o3c + M3 + 1;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  int m1 = 0, am2 = 0, am3 = 0;
  double sg2 = 1., sg3 = 1.;
  if (k < K) {
    const int4 t = km[k];
    m1 = t.x;
    am2 = abs(t.y);
    am3 = abs(t.z);
    sg2 = t.y < 0 ? -1. : 1.;
    sg3 = t.z < 0 ? -1. : 1.;
  }
  double sc = 0., ss = 0.;
  const int a0 = blockIdx.y * perPart;
  const int a1 = min(n, a0 + perPart);
  for (int t0 = a0; t0 < a1; t0 += tile) {
    const int na = min(tile, a1 - t0);
    __syncthreads();
    for (int v = threadIdx.x; v < na * W; v += blockDim.x) {
      const int e = v / na, a = v - e * na;
      const double c = tab[(size_t)e * n + t0 + a];
      // the charge goes with the first dimension's entries
      sh[a * st + e] = e < o2c ? q[t0 + a] * c : c;
    }
    __syncthreads();
    if (k < K) {
#pragma unroll 2
      for (int a = 0; a < na; ++a) {
        const double *base = sh + (size_t)a * st;
        const double c1 = base[m1], s1 = base[o1s + m1];
        const double c2 = base[o2c + am2], s2 = sg2 * base[o2s + am2];
        const double c3 = base[o3c + am3], s3 = sg3 * base[o3s + am3];
        const double cm = fma(c1, c2, -(s1 * s2));
        const double smv = fma(s1, c2, c1 * s2);
        sc = fma(-smv, s3, fma(cm, c3, sc));
        ss = fma(cm, s3, fma(smv, c3, ss));
      }
    }
  }
  if (k < K) {
    part[(size_t)(2 * blockIdx.y) * K + k] = sc;
    part[(size_t)(2 * blockIdx.y + 1) * K + k] = ss;
  }
}

// Per k: the structure factor (range sums in order), its energy term and
// virial/stress terms (src/ewald.c:300-318); S receives it times a_k, as the
// forces take it.  Block partials of {energy, stress 0..5} go to
// bpart[q * gridDim.x + block]; the last block to finish adds them, block by
// block, into sums (*done counts the blocks and returns to 0).
__global__ void k_ewald_kdata(int K, int P, const double *__restrict__ part,
                              const double4 *__restrict__ kv, const double *__restrict__ vam,
                              double2 *__restrict__ S, double *bpart, unsigned *done,
                              double *__restrict__ sums) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double v[7] = {0., 0., 0., 0., 0., 0., 0.};
  if (k < K) {
    double sc = 0., ss = 0.;
    for (int p = 0; p < P; ++p) {
      sc += part[(size_t)(2 * p) * K + k];
      ss += part[(size_t)(2 * p + 1) * K + k];
    }
    const double4 t = kv[k];
    S[k] = make_double2(t.w * sc, t.w * ss);
    double virtmp = sc * sc + ss * ss;
    v[0] = t.w * virtmp;
    virtmp *= vam[k];
    v[1] = -(virtmp * t.x * t.x);
    v[2] = -(virtmp * t.x * t.y);
    v[3] = -(virtmp * t.x * t.z);
    v[4] = -(virtmp * t.y * t.y);
    v[5] = -(virtmp * t.y * t.z);
    v[6] = -(virtmp * t.z * t.z);
  }
  __shared__ double red[7][8];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const double s = warp_sum_d(v[j]);
    if (lane == 0) red[j][w] = s;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double s = 0.;
    for (int j = 0; j < (int)(blockDim.x >> 5); ++j) s += red[threadIdx.x][j];
    bpart[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
    __threadfence();
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!last || w >= 7) return;
  __threadfence();
  double s = 0.;
  for (int b = lane; b < (int)gridDim.x; b += 32)
    s += __ldcg(bpart + (size_t)w * gridDim.x + b);
  s = warp_sum_d(s);
  if (lane == 0) sums[w] = s;
}

// Forces: one thread per atom and part of the k list (grid y): pf[3 part + c]
// [i] = q_i sum over the part's k of a_k (sin(k.r) Re S - cos(k.r) Im S) k_c.
// Along a row of fixed (m1, m2), k = base + m3 w, so the row adds base sum(d)
// + w sum(m3 d): eleven FP64 operations per k where the three components took
// eighteen.  The parts fill the SMs: one thread over the whole list was 24
// blocks for 3,000 atoms and took 0.99 ms; in 32 parts it takes 0.029.
__global__ void __launch_bounds__(128)
    k_ewald_forces(int n, int M1, int M2, int M3, int step, const int *__restrict__ rowPart,
                   const int4 *__restrict__ rows, const int *__restrict__ rowK,
                   const double4 *__restrict__ rowBase, double wx, double wy, double wz,
                   const double2 *__restrict__ S, const double *__restrict__ tab,
                   const double *__restrict__ q, double *__restrict__ pf) {
  extern __shared__ double sh[];
  const int T = blockDim.x;
  double *c3 = sh + threadIdx.x, *s3 = c3 + (size_t)(M3 + 1) * T;
  const int i = blockIdx.x * T + threadIdx.x;
  if (i >= n) return;  // no block-wide synchronisation below
  const double *c1 = tab + i, *s1 = c1 + (size_t)(M1 + 1) * n;
  const double *c2 = s1 + (size_t)(M1 + 1) * n, *s2 = c2 + (size_t)(M2 + 1) * n;
  const double *c3g = s2 + (size_t)(M2 + 1) * n, *s3g = c3g + (size_t)(M3 + 1) * n;
  for (int m = 0; m <= M3; ++m) {
    c3[m * T] = c3g[(size_t)m * n];
    s3[m * T] = s3g[(size_t)m * n];
  }
  double ax = 0., ay = 0., az = 0.;
  const int r1 = rowPart[(blockIdx.y + 1) * step];
  for (int r = rowPart[blockIdx.y * step]; r < r1; ++r) {
    const int4 row = rows[r];  // m1, m2, first m3, last m3
    const int am2 = abs(row.y);
    const double a1c = c1[(size_t)row.x * n], a1s = s1[(size_t)row.x * n];
    const double a2c = c2[(size_t)am2 * n];
    const double a2s = (row.y < 0 ? -1. : 1.) * s2[(size_t)am2 * n];
    const double cm = fma(a1c, a2c, -(a1s * a2s));
    const double smv = fma(a1s, a2c, a1c * a2s);
    const double2 *sk = S + rowK[r] - row.z;
    double A = 0., B = 0.;
#pragma unroll 4
    for (int m3 = row.z; m3 <= row.w; ++m3) {
      const int at = abs(m3) * T;
      const double t3c = c3[at], t3s = m3 < 0 ? -s3[at] : s3[at];
      const double cms = fma(cm, t3c, -(smv * t3s));
      const double sms = fma(smv, t3c, cm * t3s);
      const double2 f = sk[m3];
      const double de = fma(sms, f.x, -(cms * f.y));
      A += de;
      B = fma((double)m3, de, B);
    }
    const double4 base = rowBase[r];
    ax = fma(B, wx, fma(A, base.x, ax));
    ay = fma(B, wy, fma(A, base.y, ay));
    az = fma(B, wz, fma(A, base.z, az));
  }
  const double qi = q[i];
  double *o = pf + (size_t)3 * blockIdx.y * n + i;
  o[0] = qi * ax;
  o[n] = qi * ay;
  o[2 * (size_t)n] = qi * az;
}

// The parts in order into the forces (grid y: the component).  scaleInput:
// MDBas's ewald_rec multiplies the whole force arrays by fact0 at the end
// (src/ewald.c:335-340), f = fact0 (f_in + sum); otherwise f = f_in + fact0
// sum.
__global__ void k_ewald_add(int n, int parts, const double *__restrict__ pf, double fact0,
                            int scaleInput, double *__restrict__ fx, double *__restrict__ fy,
                            double *__restrict__ fz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double *f = (blockIdx.y == 0 ? fx : blockIdx.y == 1 ? fy : fz) + i;
  double s = 0.;
  for (int p = 0; p < parts; ++p) s += pf[((size_t)3 * p + blockIdx.y) * n + i];
  *f = scaleInput ? (*f + s) * fact0 : *f + s * fact0;
}

// The standalone calls' state (the engine keeps its own).
EwaldWork &ewald_ctx() {
  static EwaldWork c;
  return c;
}

// k list of one box / alpha / m-range, built on the host with MDBas's
// expressions (src/ewald.c:146-150, 255-300).
int build_klist(EwaldKList &kl, const PBC *box, double alpha, int M1, int M2, int M3) {
  const double key[12] = {box->u1, box->u2, box->u3, box->v1, box->v2, box->v3, box->w1,
                          box->w2, box->w3, alpha, box->u + box->v + box->w,
                          (double)M1 + 1000. * M2 + 1.e6 * M3};
  if (kl.valid && memcmp(key, kl.key, sizeof(key)) == 0) return MDBAS_NB_OK;
  kl.valid = false;
  const double rAlpha2 = -0.25 / (alpha * alpha);
  double rc = fmin(((double)M1 * box->u), ((double)M2 * box->v));
  rc = fmin(rc, (double)M3 * box->w);
  rc = rc * 1.05 * kTwoPi;
  const double rc2 = rc * rc;
  std::vector<int4> km, rows;
  std::vector<double4> kv, rowBase;
  std::vector<double> vam;
  std::vector<int> rowK;
  int m2min = 0, m3min = 1;
  for (int m1 = 0; m1 <= M1; ++m1) {
    const double rm1x = kTwoPi * box->u1 * (double)m1;
    const double rm1y = kTwoPi * box->u2 * (double)m1;
    const double rm1z = kTwoPi * box->u3 * (double)m1;
    for (int m2 = m2min; m2 <= M2; ++m2) {
      const double rm2x = rm1x + (kTwoPi * box->v1 * (double)m2);
      const double rm2y = rm1y + (kTwoPi * box->v2 * (double)m2);
      const double rm2z = rm1z + (kTwoPi * box->v3 * (double)m2);
      int lo = 0, last = 0;
      bool open = false;
      for (int m3 = m3min; m3 <= M3; ++m3) {
        const double rmx = rm2x + (kTwoPi * box->w1 * (double)m3);
        const double rmy = rm2y + (kTwoPi * box->w2 * (double)m3);
        const double rmz = rm2z + (kTwoPi * box->w3 * (double)m3);
        const double rm = rmx * rmx + rmy * rmy + rmz * rmz;
        if (rm <= rc2) {
          // in-cut-off m3 of a row are contiguous (|a + m3 b|^2 is convex in m3)
          if (open && m3 != last + 1) {
            rows.push_back(make_int4(m1, m2, lo, last));
            rowK.push_back((int)km.size() - (last - lo + 1));
            rowBase.push_back(make_double4(rm2x, rm2y, rm2z, 0.));
            open = false;
          }
          if (!open) {
            lo = m3;
            open = true;
          }
          last = m3;
          const double rrm = 1.0 / rm;
          const double am = exp(rAlpha2 * rm) * rrm;
          km.push_back(make_int4(m1, m2, m3, 0));
          kv.push_back(make_double4(rmx, rmy, rmz, am));
          vam.push_back(2.0 * am * (rrm - rAlpha2));
        }
      }
      if (open) {
        rows.push_back(make_int4(m1, m2, lo, last));
        rowK.push_back((int)km.size() - (last - lo + 1));
        rowBase.push_back(make_double4(rm2x, rm2y, rm2z, 0.));
      }
      m3min = -M3;
    }
    m2min = -M2;
  }
  // first row of each of kEwParts parts of about equally many k
  int rowPart[kEwParts + 1];
  for (int p = 0, r = 0; p <= kEwParts; ++p) {
    while (r < (int)rows.size() && (long long)rowK[r] * kEwParts < (long long)km.size() * p) ++r;
    rowPart[p] = p == kEwParts ? (int)rows.size() : r;
  }
  kl.K = (int)km.size();
  kl.nRows = (int)rows.size();
  kl.M1 = M1;
  kl.M2 = M2;
  kl.M3 = M3;
  const size_t K1 = km.empty() ? 1 : km.size(), R1 = rows.empty() ? 1 : rows.size();
  MDB_TRY(kl.km.ensure(sizeof(int4) * K1));
  MDB_TRY(kl.kv.ensure(sizeof(double4) * K1));
  MDB_TRY(kl.vam.ensure(sizeof(double) * K1));
  MDB_TRY(kl.rows.ensure(sizeof(int4) * R1));
  MDB_TRY(kl.rowK.ensure(sizeof(int) * R1));
  MDB_TRY(kl.rowBase.ensure(sizeof(double4) * R1));
  MDB_TRY(kl.rowPart.ensure(sizeof(rowPart)));
  MDB_CUDA(cudaMemcpy(kl.rowPart.p, rowPart, sizeof(rowPart), cudaMemcpyHostToDevice));
  if (kl.K) {
    MDB_CUDA(cudaMemcpy(kl.km.p, km.data(), sizeof(int4) * km.size(), cudaMemcpyHostToDevice));
    MDB_CUDA(cudaMemcpy(kl.kv.p, kv.data(), sizeof(double4) * kv.size(), cudaMemcpyHostToDevice));
    MDB_CUDA(cudaMemcpy(kl.vam.p, vam.data(), sizeof(double) * vam.size(),
                        cudaMemcpyHostToDevice));
    MDB_CUDA(cudaMemcpy(kl.rows.p, rows.data(), sizeof(int4) * rows.size(),
                        cudaMemcpyHostToDevice));
    MDB_CUDA(cudaMemcpy(kl.rowK.p, rowK.data(), sizeof(int) * rowK.size(),
                        cudaMemcpyHostToDevice));
    MDB_CUDA(cudaMemcpy(kl.rowBase.p, rowBase.data(), sizeof(double4) * rowBase.size(),
                        cudaMemcpyHostToDevice));
  }
  memcpy(kl.key, key, sizeof(key));
  kl.valid = true;
  return MDBAS_NB_OK;
}

EwBox make_ew_box(const PBC *p) {
  EwBox b;
  b.u1 = p->u1; b.u2 = p->u2; b.u3 = p->u3;
  b.v1 = p->v1; b.v2 = p->v2; b.v3 = p->v3;
  b.w1 = p->w1; b.w2 = p->w2; b.w3 = p->w3;
  return b;
}

int ewald_launch_impl(EwaldWork &c, int n, const PBC *box, double alpha, double chargeConst,
                      int M1, int M2, int M3, const double *x, const double *y, const double *z,
                      const double *q, double *fx, double *fy, double *fz, int scaleInput,
                      cudaStream_t s) {
  int dev = 0;
  MDB_CUDA(cudaGetDevice(&dev));
  if (c.device != dev) {
    c.kl.valid = false;
    c.device = dev;
  }
  MDB_TRY(build_klist(c.kl, box, alpha, M1, M2, M3));
  const EwaldKList &kl = c.kl;
  const EwBox b = make_ew_box(box);
  const int K = kl.K;
  // shared memory: the k-thread kernel's atom tile, the atom kernel's m3 table
  int maxSmem = 0;
  MDB_CUDA(cudaDeviceGetAttribute(&maxSmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t perAtom = sizeof(double) * (2 * (size_t)(M1 + M2 + M3 + 3) | 1);
  int tile = (int)((size_t)(maxSmem / 2) / perAtom);
  if (tile > 64) tile = 64;
  int fThreads = 128;
  while (fThreads > 32 && sizeof(double) * 2 * (size_t)(M3 + 1) * fThreads > (size_t)maxSmem / 2)
    fThreads /= 2;
  if (tile < 1 || sizeof(double) * 2 * (size_t)(M3 + 1) * fThreads > (size_t)maxSmem) {
    set_last_status(MDBAS_NB_ERR_UNSUPPORTED, "reciprocal m-range too large for shared memory");
    return MDBAS_NB_ERR_UNSUPPORTED;
  }
  const size_t smemF = sizeof(double) * 2 * (size_t)(M3 + 1) * fThreads;
  MDB_TRY(c.S.ensure(sizeof(double2) * (size_t)(K > 0 ? K : 1)));
  MDB_TRY(c.sums.ensure(sizeof(double) * 8));
  const double rVol = kTwoPi / box->vol;
  const double fact1 = 2.0 * rVol * chargeConst;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int parts = 0;
  if (K == 0) MDB_CUDA(cudaMemsetAsync(c.sums.p, 0, sizeof(double) * 8, s));
  if (K > 0) {
    MDB_TRY(c.tab.ensure(sizeof(double) * 2 * (size_t)(M1 + M2 + M3 + 3) * n));
    double *tab = c.tab.as<double>();
    MDB_LAUNCH(k_ewald_tables, dim3(grid_for(n, 128), 3), 128, 0, s, n, b, M1, M2, M3, x, y, z,
               tab);
    const int kBlocks = (K + kSfThreads - 1) / kSfThreads;
    int P = (4 * sms + kBlocks - 1) / kBlocks;
    P = P < 1 ? 1 : P > 32 ? 32 : P;
    if (P > n) P = n;
    const int perPart = (n + P - 1) / P;
    const size_t smemSf = perAtom * (size_t)tile;
    MDB_CUDA(cudaFuncSetAttribute(k_ewald_sf, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smemSf));
    MDB_TRY(c.part.ensure(sizeof(double) * 2 * (size_t)P * K));
    const int kdBlocks = (K + 255) / 256;
    MDB_TRY(c.bpart.ensure(sizeof(double) * 7 * (size_t)kdBlocks));
    if (!c.done.p) {
      MDB_TRY(c.done.ensure(sizeof(unsigned)));
      MDB_CUDA(cudaMemsetAsync(c.done.p, 0, sizeof(unsigned), s));
    }
    MDB_LAUNCH(k_ewald_sf, dim3(kBlocks, P), kSfThreads, smemSf, s, n, K, perPart, tile, M1, M2,
               M3, kl.km.as<int4>(), tab, q, c.part.as<double>());
    MDB_LAUNCH(k_ewald_kdata, kdBlocks, 256, 0, s, K, P, c.part.as<double>(),
               kl.kv.as<double4>(), kl.vam.as<double>(), c.S.as<double2>(),
               c.bpart.as<double>(), c.done.as<unsigned>(), c.sums.as<double>());
    // parts of the k list until there are four blocks for every SM
    const int blocks = grid_for(n, fThreads);
    parts = 1;
    while (parts < kEwParts && (long long)blocks * parts < 4 * sms) parts *= 2;
    MDB_TRY(c.pf.ensure(sizeof(double) * 3 * (size_t)parts * n));
    MDB_CUDA(cudaFuncSetAttribute(k_ewald_forces, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smemF));
    MDB_LAUNCH(k_ewald_forces, dim3(blocks, parts), fThreads, smemF, s, n, M1, M2, M3,
               kEwParts / parts, kl.rowPart.as<int>(), kl.rows.as<int4>(), kl.rowK.as<int>(),
               kl.rowBase.as<double4>(), kTwoPi * box->w1, kTwoPi * box->w2, kTwoPi * box->w3,
               c.S.as<double2>(), tab, q, c.pf.as<double>());
  }
  c.parts = parts;
  c.fact1 = fact1;
  return fx ? ewald_add(c, n, fx, fy, fz, scaleInput, s) : MDBAS_NB_OK;
}

// out[0] = energy (reciprocal + self + non-neutral), out[1] = virial,
// out[2..7] = stress, from the device sums h (src/ewald.c:323-352).
void ewald_results(double fact1, const PBC *box, double alpha, double chargeConst, double systq,
                   double sumq2, const double *h, double out[8]) {
  const double eself = -chargeConst * alpha * sumq2 / kSqrtPi;
  const double enn = -(0.5 * kPi * chargeConst) * ((systq / alpha) * (systq / alpha) / box->vol);
  const double etmp = h[0];
  double st[6];
  st[0] = fact1 * (h[1] + etmp) + enn;
  st[1] = fact1 * h[2];
  st[2] = fact1 * h[3];
  st[3] = fact1 * (h[4] + etmp) + enn;
  st[4] = fact1 * h[5];
  st[5] = fact1 * (h[6] + etmp) + enn;
  out[0] = fact1 * etmp + eself + enn;
  out[1] = -(st[0] + st[3] + st[5]);
  for (int k = 0; k < 6; ++k) out[2 + k] = st[k];
}

// Device arrays.
int ewald_run(int n, const PBC *box, double alpha, double chargeConst, int M1, int M2, int M3,
              const double *x, const double *y, const double *z, const double *q, double systq,
              double sumq2, double *fx, double *fy, double *fz, int scaleInput, double out[8],
              cudaStream_t s) {
  EwaldWork &c = ewald_ctx();
  MDB_TRY(ewald_launch_impl(c, n, box, alpha, chargeConst, M1, M2, M3, x, y, z, q, fx, fy, fz,
                            scaleInput, s));
  double h[7];
  MDB_CUDA(cudaMemcpyAsync(h, c.sums.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  MDB_CUDA(cudaStreamSynchronize(s));
  ewald_results(c.fact1, box, alpha, chargeConst, systq, sumq2, h, out);
  return MDBAS_NB_OK;
}

int nint_h(double x) { return (x >= 0.) ? (int)(x + 0.5) : (int)(x - 0.5); }

// host arrays staged through device buffers
int ewald_host(int n, const PBC *box, double alpha, double chargeConst, int M1, int M2, int M3,
               const double *x, const double *y, const double *z, const double *q, double *fx,
               double *fy, double *fz, int scaleInput, double out[8]) {
  EwaldWork &c = ewald_ctx();
  standalone_copies();
  double systq, sumq2;
  charge_sums(n, q, &systq, &sumq2);  // src/ewald.c:166-172
  cudaStream_t s = nullptr;
  MDB_TRY(c.xyzq.ensure(sizeof(double) * 4 * (size_t)n));
  MDB_TRY(c.f.ensure(sizeof(double) * 3 * (size_t)n));
  double *d = c.xyzq.as<double>(), *f = c.f.as<double>();
  const size_t bytes = sizeof(double) * (size_t)n;
  const CopySpan3 f3(fx, fy, fz, f, n);
  const CopySpan in[7] = {
      {const_cast<double *>(x), d, bytes},
      {const_cast<double *>(y), d + n, bytes, false, true},
      {const_cast<double *>(z), d + 2 * (size_t)n, bytes, false, true},
      {const_cast<double *>(q), d + 3 * (size_t)n, bytes, false, true},
      f3.s[0], f3.s[1], f3.s[2]};
  MDB_TRY(copy_in(in, 7, s));
  MDB_TRY(ewald_launch_impl(c, n, box, alpha, chargeConst, M1, M2, M3, d, d + n,
                            d + 2 * (size_t)n, d + 3 * (size_t)n, f, f + n, f + 2 * (size_t)n,
                            scaleInput, s));
  double h[7];
  const CopySpan o[4] = {f3.s[0], f3.s[1], f3.s[2], {h, c.sums.p, sizeof(h)}};
  MDB_TRY(copy_out(o, 4, s));
  ewald_results(c.fact1, box, alpha, chargeConst, systq, sumq2, h, out);
  return MDBAS_NB_OK;
}

__global__ void k_kspace_fix(const double *__restrict__ src, double scale, double add,
                             long long *__restrict__ dst) {
  if (threadIdx.x == 0 && blockIdx.x == 0) dst[0] = fix_e(scale * src[0] + add);
}

}  // namespace

int ewald_add(EwaldWork &c, int n, double *fx, double *fy, double *fz, int scaleInput,
              cudaStream_t s) {
  MDB_LAUNCH(k_ewald_add, dim3(grid_for(n, 256), 3), 256, 0, s, n, c.parts, c.pf.as<double>(),
             2.0 * c.fact1, scaleInput, fx, fy, fz);
  return MDBAS_NB_OK;
}

int ewald_launch(EwaldWork &c, int n, const PBC *box, double alpha, double chargeConst, int M1,
                 int M2, int M3, const double *x, const double *y, const double *z,
                 const double *q, double *fx, double *fy, double *fz, int scaleInput,
                 cudaStream_t s) {
  return ewald_launch_impl(c, n, box, alpha, chargeConst, M1, M2, M3, x, y, z, q, fx, fy, fz,
                           scaleInput, s);
}

void charge_sums(int n, const double *q, double *systq, double *sumq2) {
  // eight sums side by side: one chain would take four cycles an atom
  double a[8] = {}, b[8] = {};
  int i = 0;
  for (; i + 8 <= n; i += 8)
    for (int k = 0; k < 8; ++k) {
      a[k] += q[i + k];
      b[k] += q[i + k] * q[i + k];
    }
  for (int k = 0; i < n; ++i, ++k) {
    a[k] += q[i];
    b[k] += q[i] * q[i];
  }
  *systq = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
  *sumq2 = ((b[0] + b[1]) + (b[2] + b[3])) + ((b[4] + b[5]) + (b[6] + b[7]));
}

void standalone_copies() {
  static const bool entered = [] {
    host_copy_enter();
    return true;
  }();
  (void)entered;
}

int kspace_fix_launch(const double *src, double scale, double add, long long *dst,
                      cudaStream_t s) {
  MDB_LAUNCH(k_kspace_fix, 1, 32, 0, s, src, scale, add, dst);
  return MDBAS_NB_OK;
}

}  // namespace mdbas

using namespace mdbas;

extern "C" {

int mdbas_nb_ewald_rec(int nAtom, const PBC *box, double alpha, double chargeConst, int m1max,
                       int m2max, int m3max, const double *x, const double *y, const double *z,
                       const double *q, double *fx, double *fy, double *fz, double out[8],
                       int device_ptrs, void *stream) {
  if (nAtom <= 0 || !box || !x || !y || !z || !q || !fx || !fy || !fz || !out ||
      !(alpha > 0.) || m1max < 0 || m2max < 0 || m3max < 0 || !(box->vol > 0.))
    return MDBAS_NB_ERR_ARG;
  if (!device_ptrs)
    return ewald_host(nAtom, box, alpha, chargeConst, m1max, m2max, m3max, x, y, z, q, fx, fy,
                      fz, 0, out);
  std::vector<double> hq(nAtom);
  MDB_CUDA(cudaMemcpy(hq.data(), q, sizeof(double) * nAtom, cudaMemcpyDeviceToHost));
  double systq, sumq2;
  charge_sums(nAtom, hq.data(), &systq, &sumq2);
  return ewald_run(nAtom, box, alpha, chargeConst, m1max, m2max, m3max, x, y, z, q, systq, sumq2,
                   fx, fy, fz, 0, out, static_cast<cudaStream_t>(stream));
}

// MDBas's init_ewald (src/ewald.c:10-99): tolerances, alpha, the m-range and
// mmax (the number of k-vectors).  MDBas also allocates its per-atom
// tables here; the GPU keeps its own, so nothing is allocated.
void init_ewald(CTRL *ctrl, PARAM *param, EWALD *ewald, PBC *box) {
  ewald->prec = fmin(fabs(ewald->prec), 0.5);
  ewald->tol = sqrt(fabs(log(ewald->prec * param->cutOff)));
  if (!ctrl->keyAlpha)
    ewald->alpha = sqrt(fabs(log(ewald->prec * param->cutOff * ewald->tol))) / param->cutOff;
  const double ta = 2.0 * ewald->tol * ewald->alpha;
  ewald->tol1 = sqrt(-log(ewald->prec * param->cutOff * (ta * ta)));
  if (!ctrl->keyMmax) {
    ewald->m1max = nint_h(0.25 + box->pa * ewald->alpha * ewald->tol1 / kPi);
    ewald->m2max = nint_h(0.25 + box->pb * ewald->alpha * ewald->tol1 / kPi);
    ewald->m3max = nint_h(0.25 + box->pc * ewald->alpha * ewald->tol1 / kPi);
  }
  double rc = fmin(((double)ewald->m1max * box->u), ((double)ewald->m2max * box->v));
  rc = fmin(rc, (double)ewald->m3max * box->w);
  rc = rc * 1.05 * kTwoPi;
  const double rc2 = rc * rc;
  ewald->mmax = 0;
  int m2min = 0, m3min = 1;
  for (int m1 = 0; m1 <= ewald->m1max; m1++) {
    const double rm1x = kTwoPi * box->u1 * (double)m1;
    const double rm1y = kTwoPi * box->u2 * (double)m1;
    const double rm1z = kTwoPi * box->u3 * (double)m1;
    for (int m2 = m2min; m2 <= ewald->m2max; m2++) {
      const double rm2x = rm1x + (kTwoPi * box->v1 * (double)m2);
      const double rm2y = rm1y + (kTwoPi * box->v2 * (double)m2);
      const double rm2z = rm1z + (kTwoPi * box->v3 * (double)m2);
      for (int m3 = m3min; m3 <= ewald->m3max; m3++) {
        const double rmx = rm2x + (kTwoPi * box->w1 * (double)m3);
        const double rmy = rm2y + (kTwoPi * box->w2 * (double)m3);
        const double rmz = rm2z + (kTwoPi * box->w3 * (double)m3);
        if (rmx * rmx + rmy * rmy + rmz * rmz <= rc2) ewald->mmax++;
      }
      m3min = -ewald->m3max;
    }
    m2min = -ewald->m2max;
  }
}

void ewald_free(EWALD *ewald) { (void)ewald; }

// MDBas's ewald_rec (src/ewald.c:131-354) on the GPU.  As in MDBas the whole
// force arrays are multiplied by 2 fact1 after the reciprocal forces are
// added (energy() calls it first, on zeroed arrays).
double ewald_rec(PARAM *param, EWALD *ewald, PBC *box, const double x[], const double y[],
                 const double z[], double fx[], double fy[], double fz[], const double q[],
                 double stress[6], double *virEwaldRec) {
  double out[8];
  const int st = ewald_host(param->nAtom, box, ewald->alpha, param->chargeConst, ewald->m1max,
                            ewald->m2max, ewald->m3max, x, y, z, q, fx, fy, fz, 1, out);
  if (st != MDBAS_NB_OK) {
    fprintf(stderr, "ewald_rec (GPU): %s: %s\n", mdbas_nb_status_string(st),
            mdbas_nb_last_message());
    exit(1);
  }
  for (int k = 0; k < 6; ++k) stress[k] = out[2 + k];
  *virEwaldRec = out[1];
  return out[0];
}

}  // extern "C"
