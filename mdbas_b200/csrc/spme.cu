// spme.cu -- smooth particle-mesh Ewald on the GPU: MDBas's init_spme,
// spme_energy and spme_free (include/spme.h:28-40; src/spme.c) and a
// status-returning entry point.
//
// The algorithm is MDBas's (src/spme.c:357-700): per atom the cardinal
// B-splines of order nbsp and their derivatives in each dimension
// (bspgen's recursion), charges spread onto the m1 x m2 x m3 grid, an
// unnormalised e^{+i} 3-D transform (FFTW_BACKWARD), the influence function
// B(m) exp(-k^2 / 4 alpha^2) / k^2 inside the reciprocal cut-off with the
// virial, an e^{-i} transform back (FFTW_FORWARD), force interpolation with
// the mean force removed, and the energy sum(Q * (theta conv Q)) with the
// self and non-neutral terms.  The transforms are cuFFT real-to-complex and
// back (D2Z, Z2D) in the row-major layout of fftw_plan_dft_3d(m1, m2, m3),
// with the last dimension's upper half left out: the charge grid is real, and
// MDBas takes the real part of the convolved grid.  The energy sum is formed
// in reciprocal space (Parseval), where the influence function has the
// transform in hand.  Spreading, the influence function and the
// interpolation are the kernels below (FP64).
// Spreading is deterministic when every grid dimension is a multiple of 8
// (atoms binned by 8^3 grid tile, one block per tile, no atomics); other
// grids spread with FP64 atomics.
#include <cufft.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <complex>
#include <vector>

#include "host_copy.cuh"
#include "kspace.cuh"

using namespace mdbas;

namespace {

constexpr int kMaxOrder = 16;  // B-spline orders 2..16

struct SpmeBox {
  double u1, u2, u3, v1, v2, v3, w1, w2, w3;  // reciprocal vectors
  double u, v, w;                             // 1 / perpendicular widths
  double vol;
};

// B-splines and derivatives of one atom in one dimension (bspgen,
// src/spme.c:269-355): s is the scaled fractional coordinate.
template <int P>  // the order, or 0: nbspRun
__device__ __forceinline__ void bspline(double s, int nbspRun, double *bsp, double *bsd) {
  const int nbsp = P > 0 ? P : nbspRun;
  const double fr = s - trunc(s);
#pragma unroll
  for (int k = 0; k < nbsp; ++k) bsp[k] = bsd[k] = 0.;
  bsd[0] = 1.0;
  bsd[1] = -1.0;
  bsp[0] = fr;
  bsp[1] = 1.0 - fr;
#pragma unroll
  for (int k = 2; k < nbsp; ++k) {
    bsp[k] = 0.0;
#pragma unroll
    for (int j = k; j > 0; --j) {
      if (k == nbsp - 1) bsd[j] = bsp[j] - bsp[j - 1];
      const double ts = s + (double)j - trunc(s);
      bsp[j] = (ts * bsp[j] + ((double)(k + 1) - ts) * bsp[j - 1]) * (1.0 / (double)k);
    }
    if (k == nbsp - 1) bsd[0] = bsp[0];
    bsp[0] = fr * bsp[0] * (1.0 / (double)k);
  }
}

// grid index of the stencil point base cell - offset; base cells are stored
// in [0, m), so one wrap brings it into [0, m) as MDBas's does for atoms in
// the box (src/spme.c:453-481)
__device__ __forceinline__ int wrap_index(int i, int m) { return i < 0 ? i + m : i; }

// base cell in [0, m).  MDBas's (int)s lies in [0, m] for atoms in the box
// (image_update wraps them there before every energy call) and its indices
// (int)s - a wrap to the same grid points; for atoms further out the
// periodic image is used, which keeps every grid access in bounds (MDBas
// folds indices >= m onto plane 0 and leaves the array below -(m - p + 1)).
__device__ __forceinline__ int cell_mod(int c, int m) {
  c %= m;
  return c < 0 ? c + m : c;
}

constexpr int kSpTile = 8;  // grid tile edge of the deterministic spreading

// Per atom and dimension (one thread each): the grid coordinate, B-splines
// (bsp[3][nbsp], bsd[3][nbsp] per atom) and the integer grid cell.  With tiles
// (tileOf not null) also the tile of the atom's base cell and the tiles'
// counts.  Blocks of 96 threads hold whole atoms.
constexpr int kSplThreads = 96;
template <int P>  // the order, or 0: nbspRun
__global__ void __launch_bounds__(kSplThreads)
    k_spme_splines(int n, SpmeBox b, int m1, int m2, int m3, int nbspRun,
                   const double *__restrict__ x, const double *__restrict__ y,
                   const double *__restrict__ z, double *__restrict__ spl,
                   int *__restrict__ cell, int *__restrict__ tileOf, int *__restrict__ count) {
  __shared__ int sc[kSplThreads];
  const int nbsp = P > 0 ? P : nbspRun;
  const int t = blockIdx.x * kSplThreads + threadIdx.x;
  if (t < 3 * n) {
    const int i = t / 3, d = t - 3 * (t / 3);
    double s;
    if (d == 0) s = (double)m1 * (x[i] * b.u1 + y[i] * b.u2 + z[i] * b.u3 + 0.5);
    else if (d == 1) s = (double)m2 * (x[i] * b.v1 + y[i] * b.v2 + z[i] * b.v3 + 0.5);
    else s = (double)m3 * (x[i] * b.w1 + y[i] * b.w2 + z[i] * b.w3 + 0.5);
    double *o = spl + (size_t)i * 6 * nbsp;
    double bp[P > 0 ? P : kMaxOrder], bd[P > 0 ? P : kMaxOrder];
    bspline<P>(s, nbsp, bp, bd);
#pragma unroll
    for (int k = 0; k < (P > 0 ? P : nbsp); ++k) {
      o[d * nbsp + k] = bp[k];
      o[(3 + d) * nbsp + k] = bd[k];
    }
    const int c = cell_mod((int)s, d == 0 ? m1 : (d == 1 ? m2 : m3));
    cell[3 * i + d] = c;
    sc[threadIdx.x] = c / kSpTile;
  }
  if (!tileOf) return;
  __syncthreads();
  const int a = blockIdx.x * (kSplThreads / 3) + threadIdx.x;
  if (threadIdx.x < kSplThreads / 3 && a < n) {
    const int *c = sc + 3 * threadIdx.x;
    const int tile = (c[0] * (m2 / kSpTile) + c[1]) * (m3 / kSpTile) + c[2];
    tileOf[a] = tile;
    atomicAdd(count + tile, 1);
  }
}

// Charge spreading: one thread per (atom, first-dimension offset).
__global__ void k_spme_spread(int n, int m1, int m2, int m3, int nbsp,
                              const double *__restrict__ q, const double *__restrict__ spl,
                              const int *__restrict__ cell, double *__restrict__ qsp) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n * nbsp) return;
  const int l = (int)(t / nbsp), a = (int)(t % nbsp);
  const double *o = spl + (size_t)l * 6 * nbsp;
  const int ii = wrap_index(cell[3 * l] - a, m1);
  const double qa = q[l] * o[a];
  for (int bb = 0; bb < nbsp; ++bb) {
    const int jj = wrap_index(cell[3 * l + 1] - bb, m2);
    const double qab = qa * o[nbsp + bb];
    const size_t base = (size_t)m3 * (jj + (size_t)m2 * ii);
    for (int c = 0; c < nbsp; ++c) {
      const int kk = wrap_index(cell[3 * l + 2] - c, m3);
      atomicAdd(qsp + base + kk, qab * o[2 * nbsp + c]);
    }
  }
}

// Deterministic spreading.  The grid is cut into 8^3 tiles (every grid
// dimension a multiple of 8); atoms are binned by the tile of their base
// cell and each bin is put in ascending atom order.  Phase one, one block per
// tile: the bin's atoms, one after the other, scatter their p^3 stencils
// into a shared-memory copy of the tile plus its halo ((8 + p - 1)^3 points:
// a stencil reaches p - 1 cells below its base cell), one thread per stencil
// point; the halo boxes go to global memory.  Phase two, one thread per grid
// point: the sum over the halo boxes that cover the point (its own tile and
// the next ones upward, as far as the order reaches) in a fixed order.  No
// atomics: the same sums in the same order on every run.
constexpr int kSpBatch = 32;
constexpr int kSpPts = (kMaxOrder * kMaxOrder * kMaxOrder + 511) / 512;  // per thread

// Exclusive scan of the tiles' counts, one block; the fill marks cleared.
__global__ void __launch_bounds__(1024)
    k_spme_tile_scan(int nt, const int *__restrict__ count, int *__restrict__ start,
                     int *__restrict__ fill) {
  __shared__ int wsum[32];
  __shared__ int carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  for (int base = 0; base < nt; base += 4096) {
    __syncthreads();
    int v[4], sum = 0;
    const int at = base + 4 * threadIdx.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = at + k < nt ? count[at + k] : 0;
      sum += v[k];
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
      int s = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      wsum[lane] = s;
    }
    __syncthreads();
    int run = carry + x - sum + (w > 0 ? wsum[w - 1] : 0);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (at + k < nt) {
        start[at + k] = run;
        fill[at + k] = 0;
        run += v[k];
      }
    __syncthreads();
    if (threadIdx.x == 0) carry += wsum[31];
  }
  __syncthreads();
  if (threadIdx.x == 0) start[nt] = carry;
}

__global__ void k_spme_tile_fill(int n, const int *__restrict__ tileOf,
                                 const int *__restrict__ start, int *__restrict__ fill,
                                 int *__restrict__ list) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int t = tileOf[i];
  list[start[t] + atomicAdd(fill + t, 1)] = i;
}

// one block per bin: its atoms in ascending index order (rank sort)
__global__ void k_spme_tile_sort(const int *__restrict__ start, const int *__restrict__ list,
                                 int *__restrict__ sorted) {
  const int s0 = start[blockIdx.x], s1 = start[blockIdx.x + 1];
  for (int u = s0 + threadIdx.x; u < s1; u += blockDim.x) {
    const int a = list[u];
    int rank = 0;
    for (int v = s0; v < s1; ++v) rank += list[v] < a;
    sorted[s0 + rank] = a;
  }
}

template <int PTS>  // stencil points per thread: 1 when p^3 <= 512
__global__ void __launch_bounds__(512, PTS == 1 ? 3 : 2)
    k_spme_spread_halo(int nbsp, int nt2, int nt3, const double *__restrict__ q,
                       const double *__restrict__ spl, const int *__restrict__ cell,
                       const int *__restrict__ start, const int *__restrict__ sorted,
                       double *__restrict__ halo) {
  extern __shared__ double hb[];  // (8 + p - 1)^3 halo box
  __shared__ double sq[kSpBatch];
  __shared__ int sc[kSpBatch];
  __shared__ double sb[kSpBatch][3 * kMaxOrder];
  const int tile = blockIdx.x;
  const int t3 = tile % nt3, t2 = (tile / nt3) % nt2, t1 = tile / (nt2 * nt3);
  const int H = kSpTile + nbsp - 1, H3 = H * H * H, p3 = nbsp * nbsp * nbsp;
  const int th = threadIdx.x;
  // this thread's stencil points (a, b, c), at most PTS of them
  int abc[PTS];
#pragma unroll
  for (int k = 0; k < PTS; ++k) {
    const int idx = th + k * 512;
    abc[k] = idx / (nbsp * nbsp) | ((idx / nbsp) % nbsp) << 8 | (idx % nbsp) << 16;
  }
  for (int u = th; u < H3; u += blockDim.x) hb[u] = 0.;
  const int s0 = start[tile], s1 = start[tile + 1];
  for (int base = s0; base < s1; base += kSpBatch) {
    const int cnt = min(kSpBatch, s1 - base);
    __syncthreads();
    if (th < cnt) {
      const int a = sorted[base + th];
      sq[th] = q[a];
      // the stencil's top corner in the halo box: base cell - tile origin + p - 1
      sc[th] = ((cell[3 * a] - kSpTile * t1 + nbsp - 1) * H +
                (cell[3 * a + 1] - kSpTile * t2 + nbsp - 1)) * H +
               (cell[3 * a + 2] - kSpTile * t3 + nbsp - 1);
    }
    for (int idx = th; idx < cnt * 3 * nbsp; idx += blockDim.x) {
      const int u = idx / (3 * nbsp), r = idx - u * 3 * nbsp;
      sb[u][r] = spl[(size_t)sorted[base + u] * 6 * nbsp + r];
    }
    __syncthreads();
    for (int u = 0; u < cnt; ++u) {
      const double qu = sq[u];
      const int su = sc[u];
#pragma unroll
      for (int k = 0; k < PTS; ++k)
        if (th + k * 512 < p3) {
          const int a = abc[k] & 0xff, bb = (abc[k] >> 8) & 0xff, c = abc[k] >> 16;
          hb[su - (a * H + bb) * H - c] +=
              ((qu * sb[u][a]) * sb[u][nbsp + bb]) * sb[u][2 * nbsp + c];
        }
      __syncthreads();  // the next atom may hit the same points
    }
  }
  __syncthreads();
  double *out = halo + (size_t)tile * H3;
  for (int u = th; u < H3; u += blockDim.x) out[u] = hb[u];
}

// Phase one for a B-spline order P known at compile time (P <= 9, so the
// (8 + P - 1)^2 rows of the halo box fit one block): each thread owns one
// row (l1, l2) of the box in registers; an atom covers the row when its
// stencil planes reach l1 and l2, and then adds ((q b1_a) b2_b) b3_c to the
// row's points -- the same products, summed over the bin's atoms in the same
// ascending order, as k_spme_spread_halo, but no thread ever touches
// another's row: no barrier per atom.  The z weights are staged with zeros on
// both sides, so every point of the row takes one broadcast load and one FMA
// at a fixed register, where a row in shared memory took a load and a store
// beside them (97 -> 79 us at 96,000 atoms, 128^3, order 8).  The block
// also puts its bin in ascending order (rank sort) for the interpolation.
template <int P>
__global__ void __launch_bounds__(256)
    k_spme_spread_rows(int nt2, int nt3, const double *__restrict__ q,
                       const double *__restrict__ spl, const int *__restrict__ cell,
                       const int *__restrict__ start, const int *__restrict__ list,
                       int *sorted, double *__restrict__ halo) {
  constexpr int H = kSpTile + P - 1, H3 = H * H * H;
  static_assert(H * H <= 256, "one row per thread");
  constexpr int kPad = kSpTile - 1, kZ = P + 2 * kPad;
  __shared__ double hb[H3];
  __shared__ int sx[kSpBatch], sy[kSpBatch], sz[kSpBatch];
  __shared__ double sb[kSpBatch][2 * P];  // q b1, b2
  __shared__ double sbz[kSpBatch][kZ];    // b3 between zeros
  const int tile = blockIdx.x;
  const int t3 = tile % nt3, t2 = (tile / nt3) % nt2, t1 = tile / (nt2 * nt3);
  const int th = threadIdx.x;
  const bool mine = th < H * H;
  const int l1 = th / H, l2 = th - (th / H) * H;
  const int s0 = start[tile], s1 = start[tile + 1];
  for (int u = s0 + th; u < s1; u += blockDim.x) {
    const int a = list[u];
    int rank = 0;
    for (int v = s0; v < s1; ++v) rank += list[v] < a;
    sorted[s0 + rank] = a;
  }
  double acc[H];
#pragma unroll
  for (int k = 0; k < H; ++k) acc[k] = 0.;
  for (int u = th; u < kSpBatch * kZ; u += blockDim.x) (&sbz[0][0])[u] = 0.;
  for (int base = s0; base < s1; base += kSpBatch) {
    const int cnt = min(kSpBatch, s1 - base);
    __syncthreads();
    if (th < cnt) {
      const int a = sorted[base + th];
      // the stencil's top corner in the halo box: base cell - tile origin + P - 1
      sx[th] = cell[3 * a] - kSpTile * t1 + P - 1;
      sy[th] = cell[3 * a + 1] - kSpTile * t2 + P - 1;
      sz[th] = cell[3 * a + 2] - kSpTile * t3 + P - 1;
    }
    for (int idx = th; idx < cnt * 3 * P; idx += blockDim.x) {
      const int u = idx / (3 * P), r = idx - u * 3 * P;
      const int a = sorted[base + u];
      const double v = spl[(size_t)a * 6 * P + r];
      if (r < P) sb[u][r] = q[a] * v;
      else if (r < 2 * P) sb[u][r] = v;
      else sbz[u][kPad + r - 2 * P] = v;
    }
    __syncthreads();
    if (mine)
      for (int u = 0; u < cnt; ++u) {
        const int a = sx[u] - l1, bb = sy[u] - l2;
        if ((unsigned)a < (unsigned)P && (unsigned)bb < (unsigned)P) {
          const double w = sb[u][a] * sb[u][P + bb];
          const double *bz = &sbz[u][kPad + sz[u]];  // point k takes b3[sz - k]
#pragma unroll
          for (int k = 0; k < H; ++k) acc[k] += w * bz[-k];
        }
      }
  }
  if (mine) {
#pragma unroll
    for (int k = 0; k < H; ++k) hb[th * H + k] = acc[k];
  }
  __syncthreads();
  double *out = halo + (size_t)tile * H3;
  for (int u = th; u < H3; u += blockDim.x) out[u] = hb[u];
}

// Phase two: grid point g takes, per dimension, the halo boxes of tiles
// tg + d (d = 0 .. reach - 1, modulo the tile count) at the local coordinate
// g - 8 (tg + d) + p - 1 when that is >= 0.  Grid (ceil(m2 m3 / blockDim), m1), plane i =
// blockIdx.y.
__global__ void k_spme_halo_gather(int m1, int m2, int m3, int nbsp, int reach, int nt1,
                                   int nt2, int nt3, const double *__restrict__ halo,
                                   double *__restrict__ qsp) {
  const int i = blockIdx.y;
  const int t2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (t2 >= m2 * m3) return;
  const long long t = (long long)i * m2 * m3 + t2;
  const int j = t2 / m3, k = t2 - j * m3;
  const int H = kSpTile + nbsp - 1, H3 = H * H * H;
  const int ti = i / kSpTile, tj = j / kSpTile, tk = k / kSpTile;
  double acc = 0.;
  for (int d1 = 0; d1 < reach; ++d1) {
    const int l1 = i - kSpTile * (ti + d1) + nbsp - 1;
    if (l1 < 0) break;
    const int s1 = (ti + d1) % nt1;
    for (int d2 = 0; d2 < reach; ++d2) {
      const int l2 = j - kSpTile * (tj + d2) + nbsp - 1;
      if (l2 < 0) break;
      const int s2 = (tj + d2) % nt2;
      for (int d3 = 0; d3 < reach; ++d3) {
        const int l3 = k - kSpTile * (tk + d3) + nbsp - 1;
        if (l3 < 0) break;
        const int s3 = (tk + d3) % nt3;
        const size_t src = ((size_t)s1 * nt2 + s2) * nt3 + s3;
        acc += halo[src * H3 + ((size_t)l1 * H + l2) * H + l3];
      }
    }
  }
  qsp[t] = acc;
}

// The same for orders P <= 9 (two halo boxes per dimension at most), fully
// unrolled: same terms, same order.
template <int P>
__global__ void k_spme_halo_gather2(int m2, int m3, int nt1, int nt2, int nt3,
                                    const double *__restrict__ halo, double *__restrict__ qsp) {
  constexpr int H = kSpTile + P - 1, H3 = H * H * H;
  static_assert(P <= 9, "two halo boxes per dimension");
  const int i = blockIdx.y;
  const int t2 = blockIdx.x * blockDim.x + threadIdx.x;
  if (t2 >= m2 * m3) return;
  const long long t = (long long)i * m2 * m3 + t2;
  const int j = t2 / m3, k = t2 - j * m3;
  const int ti = i / kSpTile, tj = j / kSpTile, tk = k / kSpTile;
  // local coordinates in the own tile's box (d = 0) and the next one (d = 1)
  const int l1 = i - kSpTile * ti + P - 1, l2 = j - kSpTile * tj + P - 1,
            l3 = k - kSpTile * tk + P - 1;
  const int u1 = ti + 1 == nt1 ? 0 : ti + 1, u2 = tj + 1 == nt2 ? 0 : tj + 1,
            u3 = tk + 1 == nt3 ? 0 : tk + 1;
  const bool n1 = l1 >= kSpTile, n2 = l2 >= kSpTile, n3 = l3 >= kSpTile;
  double acc = 0.;
#pragma unroll
  for (int d1 = 0; d1 < 2; ++d1) {
    if (d1 == 1 && !n1) break;
    const int s1 = d1 ? u1 : ti, m1l = l1 - kSpTile * d1;
#pragma unroll
    for (int d2 = 0; d2 < 2; ++d2) {
      if (d2 == 1 && !n2) break;
      const int s2 = d2 ? u2 : tj, m2l = l2 - kSpTile * d2;
#pragma unroll
      for (int d3 = 0; d3 < 2; ++d3) {
        if (d3 == 1 && !n3) break;
        const int s3 = d3 ? u3 : tk, m3l = l3 - kSpTile * d3;
        const size_t src = ((size_t)s1 * nt2 + s2) * nt3 + s3;
        acc += halo[src * H3 + (m1l * H + m2l) * H + m3l];
      }
    }
  }
  qsp[t] = acc;
}

// Sums over all blocks, run-to-run identical: each block's sums of v[0..N) go
// to part[c * blocks + id] by a fixed tree, and the last block to finish adds
// the blocks' partials in a fixed order into dst (*done counts the blocks and
// returns to 0).  Called by every thread of blocks of 256.
template <int N>
__device__ __forceinline__ void grid_sum(const double (&v)[N], double *part, int id, int blocks,
                                         unsigned *done, double *__restrict__ dst) {
  __shared__ double red[N][8];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    const double s = warp_sum_d(v[c]);
    if (lane == 0) red[c][w] = s;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double s = 0.;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[threadIdx.x][k];
    part[(size_t)threadIdx.x * blocks + id] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(done, blocks - 1) == (unsigned)(blocks - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll 1
  for (int c = 0; c < N; ++c) {
    double s = 0.;
    for (int k = threadIdx.x; k < blocks; k += 256) s += __ldcg(part + (size_t)c * blocks + k);
    s = warp_sum_d(s);
    if (lane == 0) red[c][w] = s;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double s = 0.;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[threadIdx.x][k];
    dst[threadIdx.x] = s;
  }
}

// A reciprocal grid point's influence value and k vector (src/spme.c:
// 460-530); 0 outside the cut-off and at the origin.
struct KPoint {
  double a, x, y, z, rrm;
};
__device__ __forceinline__ KPoint k_point(const SpmeBox &b, int ii, int jj, int kk, double bm,
                                          double ralpha2, double rc2) {
  const double tw = 6.283185307179586;
  const double ti = tw * (double)ii, tj = tw * (double)jj, tk = tw * (double)kk;
  KPoint p;
  p.x = ti * b.u1 + tj * b.v1 + tk * b.w1;
  p.y = ti * b.u2 + tj * b.v2 + tk * b.w2;
  p.z = ti * b.u3 + tj * b.v3 + tk * b.w3;
  const double rm = p.x * p.x + p.y * p.y + p.z * p.z;
  const bool in = rm > 2.220446049250313e-16 && rm <= rc2;
  p.rrm = in ? 1.0 / rm : 0.;
  p.a = in ? bm * exp(ralpha2 * rm) * p.rrm : 0.;
  return p;
}

// Influence function, virial and energy on the half grid m1 x m2 x (m3/2 + 1).
// Each point stands for itself and, inside the half (0 < k, 2k < m3), for the
// point at the negative indices that the real transform leaves out.  That
// point's k vector is the negative one except in the planes at half a grid
// length, whose index MDBas takes as +m/2 on both sides: there it is
// evaluated on its own.  The transform back is of the real part, so the grid
// is multiplied by the two points' mean.  sums[0..5] stress, sums[6] energy.
// Plane i = blockIdx.y; blocks of 256 stride over it.  128^3: 27 us where the
// full complex grid took 38, the energy's own pass over both grids 12 and the
// separate sums 18.
__global__ void __launch_bounds__(256)
    k_spme_influence(int m1, int m2, int m3, SpmeBox b, double ralpha2, double rc2,
                     const double *__restrict__ bmod,  // m1 + m2 + m3
                     cufftDoubleComplex *__restrict__ ft, double *part, unsigned *done,
                     double *__restrict__ sums) {
  const int i = blockIdx.y, mh = m3 / 2 + 1;
  const int ii = i > m1 / 2 ? i - m1 : i;
  double s[7] = {0., 0., 0., 0., 0., 0., 0.};
  for (int t2 = blockIdx.x * 256 + threadIdx.x; t2 < m2 * mh; t2 += gridDim.x * 256) {
    const int j = t2 / mh, k = t2 - j * mh;
    const int jj = j > m2 / 2 ? j - m2 : j;
    const double bm = bmod[i] * bmod[m1 + j] * bmod[m1 + m2 + k];
    const KPoint p = k_point(b, ii, jj, k, bm, ralpha2, rc2);
    const bool two = k > 0 && 2 * k < m3;
    KPoint c = p;
    if (2 * i == m1 || 2 * j == m2 || 2 * k == m3)
      c = k_point(b, 2 * i == m1 ? ii : -ii, 2 * j == m2 ? jj : -jj, 2 * k == m3 ? k : -k, bm,
                  ralpha2, rc2);
    const size_t t = (size_t)i * m2 * mh + t2;
    cufftDoubleComplex f = ft[t];
    const double f2 = f.x * f.x + f.y * f.y;
    const double e = p.a * f2, e2 = two ? c.a * f2 : 0.;
    const double v = 2.0 * (p.rrm - ralpha2) * e, v2 = 2.0 * (c.rrm - ralpha2) * e2;
    s[0] -= v * p.x * p.x + v2 * c.x * c.x;
    s[1] -= v * p.x * p.y + v2 * c.x * c.y;
    s[2] -= v * p.x * p.z + v2 * c.x * c.z;
    s[3] -= v * p.y * p.y + v2 * c.y * c.y;
    s[4] -= v * p.y * p.z + v2 * c.y * c.z;
    s[5] -= v * p.z * p.z + v2 * c.z * c.z;
    s[6] += e + e2;
    const double a = 0.5 * (p.a + c.a);
    f.x *= a;
    f.y *= a;
    ft[t] = f;
  }
  grid_sum<7>(s, part, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y, done, sums);
}

// Force interpolation (src/spme.c:532-575) into fr[3][n]; sums for the mean.
// MDBas's triple sum over the p^3 grid points of an atom factorises:
//   sum_abc Q(a,b,c) d1_a b2_b b3_c = sum_a d1_a sum_b b2_b sum_c Q b3_c
// (likewise for the y and z parts), so per (a, b) row only the two sums
// over c of Q b3_c and Q d3_c are needed.  `group` lanes (the next power of
// two >= p) share one atom, lane a taking the plane a; the group's three
// partial forces are summed with shuffles.
__global__ void __launch_bounds__(256)
    k_spme_forces(int n, int m1, int m2, int m3, int nbsp, int group, SpmeBox b,
                              double fact1, const double *__restrict__ q,
                              const double *__restrict__ spl, const int *__restrict__ cell,
                              const double *__restrict__ conv, double *__restrict__ fr,
                              double *part, unsigned *done, double *__restrict__ fsum) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int l = (int)(t / group), a = (int)(t % group);
  double px = 0., py = 0., pz = 0.;
  if (l < n && a < nbsp) {
    const double *o = spl + (size_t)l * 6 * nbsp;
    const double *b2 = o + nbsp, *b3 = o + 2 * nbsp;
    const double *d2 = o + 4 * nbsp, *d3 = o + 5 * nbsp;
    const int ii = wrap_index(cell[3 * l] - a, m1);
    const int cy = cell[3 * l + 1], cz = cell[3 * l + 2];
    double t1 = 0., t2 = 0., t3 = 0.;
    for (int bb = 0; bb < nbsp; ++bb) {
      const int jj = wrap_index(cy - bb, m2);
      const size_t base = (size_t)m3 * (jj + (size_t)m2 * ii);
      double sb = 0., sd = 0.;
      for (int c = 0; c < nbsp; ++c) {
        const double qt = conv[base + wrap_index(cz - c, m3)];
        sb += qt * __ldg(b3 + c);
        sd += qt * __ldg(d3 + c);
      }
      const double wb = __ldg(b2 + bb);
      t1 += wb * sb;
      t2 += __ldg(d2 + bb) * sb;
      t3 += wb * sd;
    }
    px = __ldg(o + 3 * nbsp + a) * t1;  // d1_a
    const double b1a = __ldg(o + a);
    py = b1a * t2;
    pz = b1a * t3;
  }
  for (int off = group >> 1; off > 0; off >>= 1) {
    px += __shfl_xor_sync(0xffffffffu, px, off);
    py += __shfl_xor_sync(0xffffffffu, py, off);
    pz += __shfl_xor_sync(0xffffffffu, pz, off);
  }
  double fx = 0., fy = 0., fz = 0.;
  if (l < n && a == 0) {
    const double fbx = px * (double)m1, fby = py * (double)m2, fbz = pz * (double)m3;
    const double fq = fact1 * q[l];
    fx = fq * (fbx * b.u1 + fby * b.v1 + fbz * b.w1);
    fy = fq * (fbx * b.u2 + fby * b.v2 + fbz * b.w2);
    fz = fq * (fbx * b.u3 + fby * b.v3 + fbz * b.w3);
    fr[l] = fx;
    fr[n + l] = fy;
    fr[2 * (size_t)n + l] = fz;
  }
  const double f[3] = {fx, fy, fz};
  grid_sum<3>(f, part, blockIdx.x, gridDim.x, done, fsum);
}

// Force interpolation per grid tile (same arithmetic per atom as
// k_spme_forces): the block loads the tile's halo box of the convolved grid
// (local l is grid point 8 t - (p - 1) + l modulo m) into shared
// memory, then takes the bin's atoms, `group` lanes per atom.  fsum gets one
// partial per tile, accumulated in atom order.
template <int P>  // the B-spline order, or 0: given at run time
__global__ void __launch_bounds__(256, 4)  // four blocks per SM (64 registers)
    k_spme_forces_tiled(int n, int m1, int m2, int m3, int nbspRun, int group, int nt2, int nt3,
                        SpmeBox b, double fact1, const double *__restrict__ q,
                        const double *__restrict__ spl, const int *__restrict__ cell,
                        const int *__restrict__ start, const int *__restrict__ sorted,
                        const double *__restrict__ conv, double *__restrict__ fr, double *part,
                        unsigned *done, double *__restrict__ fsum) {
  extern __shared__ double hb[];
  const int nbsp = P > 0 ? P : nbspRun;
  const int tile = blockIdx.x;
  const int t3 = tile % nt3, t2 = (tile / nt3) % nt2, t1 = tile / (nt2 * nt3);
  const int H = kSpTile + nbsp - 1;
  // the box point by point, all of a thread's copies in flight at once and the
  // point's place carried along (a warp per row, 15 of its lanes at work, four
  // rows in flight: 95 us at 96,000 atoms, 128^3, order 8; this 75)
  const int o1 = kSpTile * t1 - (nbsp - 1), o2 = kSpTile * t2 - (nbsp - 1),
            o3 = kSpTile * t3 - (nbsp - 1);
  const int H2 = H * H, H3 = H2 * H;
  const int e1 = 256 / H2, e2 = 256 % H2 / H, e3 = 256 % H;  // 256 points further
  int l1 = (int)threadIdx.x / H2, l2 = (int)threadIdx.x % H2 / H, l3 = (int)threadIdx.x % H;
#pragma unroll 4
  for (int u = threadIdx.x; u < H3; u += 256) {
    const int g1 = o1 + l1 < 0 ? o1 + l1 + m1 : o1 + l1;
    const int g2 = o2 + l2 < 0 ? o2 + l2 + m2 : o2 + l2;
    const int g3 = o3 + l3 < 0 ? o3 + l3 + m3 : o3 + l3;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(hb + u)),
                 "l"(conv + (((size_t)g1 * m2 + g2) * m3 + g3))
                 : "memory");
    l1 += e1;
    l2 += e2;
    l3 += e3;
    if (l3 >= H) {
      l3 -= H;
      ++l2;
    }
    if (l2 >= H) {
      l2 -= H;
      ++l1;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int s0 = start[tile], s1 = start[tile + 1];
  const int per = blockDim.x / group, a = threadIdx.x % group;
  double sx = 0., sy = 0., sz = 0.;
  for (int base = s0; base < s1; base += per) {  // same trip count in the whole block
    const int u = base + (int)threadIdx.x / group;
    const int l = u < s1 ? sorted[u] : -1;
    double px = 0., py = 0., pz = 0.;
    if (l >= 0 && a < nbsp) {
      const double *o = spl + (size_t)l * 6 * nbsp;
      const double *b2 = o + nbsp, *b3 = o + 2 * nbsp;
      const double *d2 = o + 4 * nbsp, *d3 = o + 5 * nbsp;
      const int c1 = cell[3 * l] - kSpTile * t1 + nbsp - 1 - a;  // plane a, local
      const int cy = cell[3 * l + 1] - kSpTile * t2 + nbsp - 1;
      const int cz = cell[3 * l + 2] - kSpTile * t3 + nbsp - 1;
      double t1s = 0., t2s = 0., t3s = 0.;
      if constexpr (P > 0) {
        double rb3[P], rd3[P];
#pragma unroll
        for (int c = 0; c < P; ++c) {
          rb3[c] = __ldg(b3 + c);
          rd3[c] = __ldg(d3 + c);
        }
#pragma unroll
        for (int bb = 0; bb < P; ++bb) {
          const double *row = hb + (c1 * H + cy - bb) * H + cz;
          double sb = 0., sd = 0.;
#pragma unroll
          for (int c = 0; c < P; ++c) {
            const double qt = row[-c];
            sb += qt * rb3[c];
            sd += qt * rd3[c];
          }
          const double wb = __ldg(b2 + bb);
          t1s += wb * sb;
          t2s += __ldg(d2 + bb) * sb;
          t3s += wb * sd;
        }
      } else {
        for (int bb = 0; bb < nbsp; ++bb) {
          const double *row = hb + (c1 * H + cy - bb) * H + cz;
          double sb = 0., sd = 0.;
          for (int c = 0; c < nbsp; ++c) {
            const double qt = row[-c];
            sb += qt * __ldg(b3 + c);
            sd += qt * __ldg(d3 + c);
          }
          const double wb = __ldg(b2 + bb);
          t1s += wb * sb;
          t2s += __ldg(d2 + bb) * sb;
          t3s += wb * sd;
        }
      }
      px = __ldg(o + 3 * nbsp + a) * t1s;  // d1_a
      const double b1a = __ldg(o + a);
      py = b1a * t2s;
      pz = b1a * t3s;
    }
    for (int o = group >> 1; o > 0; o >>= 1) {
      px += __shfl_xor_sync(0xffffffffu, px, o);
      py += __shfl_xor_sync(0xffffffffu, py, o);
      pz += __shfl_xor_sync(0xffffffffu, pz, o);
    }
    if (l >= 0 && a == 0) {
      const double fbx = px * (double)m1, fby = py * (double)m2, fbz = pz * (double)m3;
      const double fq = fact1 * q[l];
      const double fx = fq * (fbx * b.u1 + fby * b.v1 + fbz * b.w1);
      const double fy = fq * (fbx * b.u2 + fby * b.v2 + fbz * b.w2);
      const double fz = fq * (fbx * b.u3 + fby * b.v3 + fbz * b.w3);
      fr[l] = fx;
      fr[n + l] = fy;
      fr[2 * (size_t)n + l] = fz;
      sx += fx;
      sy += fy;
      sz += fz;
    }
  }
  const double f[3] = {sx, sy, sz};
  grid_sum<3>(f, part, blockIdx.x, gridDim.x, done, fsum);
}

// f += fr - mean (device arrays)
__global__ void k_spme_add(int n, const double *__restrict__ fr, const double *__restrict__ fsum,
                           double *__restrict__ fx, double *__restrict__ fy,
                           double *__restrict__ fz) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n) return;
  const double inv = 1.0 / (double)n;
  fx[l] += fr[l] - fsum[0] * inv;
  fy[l] += fr[n + l] - fsum[1] * inv;
  fz[l] += fr[2 * (size_t)n + l] - fsum[2] * inv;
}

// |bspc|^2 of one dimension (epl_cplx/bspcoef, src/spme.c:170-267).
void bsp_moduli(int m, int nbsp, double *out) {
  std::vector<double> bsp(nbsp, 0.0);
  bsp[1] = 1.0;
  for (int k = 2; k < nbsp; ++k) {
    bsp[k] = 0.0;
    for (int j = k; j > 0; --j) bsp[j] = ((double)j * bsp[j] + (double)(k + 1 - j) * bsp[j - 1]) / k;
  }
  std::vector<std::complex<double>> epl(m);
  epl[0] = 1.0;
  for (int i = 1; i <= m / 2; ++i) {
    epl[i] = std::exp(std::complex<double>(0.0, 6.283185307179586 * (double)i / (double)m));
    epl[m - i] = std::conj(epl[i]);
  }
  for (int i = 0; i < m; ++i) {
    std::complex<double> coeff(0.0, 0.0);
    for (int k = 0; k < nbsp - 1; ++k) coeff += bsp[k + 1] * epl[(size_t)((long long)i * k % m)];
    const std::complex<double> c = epl[(size_t)((long long)i * (nbsp - 1) % m)] / coeff;
    out[i] = std::real(c * std::conj(c));
  }
}

// The standalone calls' state (the engine keeps its own).
SpmeWork &spme_ctx() {
  static SpmeWork c;
  return c;
}

SpmeBox make_spme_box(const PBC *p) {
  SpmeBox b;
  b.u1 = p->u1; b.u2 = p->u2; b.u3 = p->u3;
  b.v1 = p->v1; b.v2 = p->v2; b.v3 = p->v3;
  b.w1 = p->w1; b.w2 = p->w2; b.w3 = p->w3;
  b.u = p->u; b.v = p->v; b.w = p->w;
  b.vol = p->vol;
  return b;
}

int cufft_check(cufftResult r, const char *what) {
  if (r == CUFFT_SUCCESS) return MDBAS_NB_OK;
  char buf[128];
  snprintf(buf, sizeof(buf), "%s failed (cufftResult %d)", what, (int)r);
  set_last_status(MDBAS_NB_ERR_CUDA, buf);
  return MDBAS_NB_ERR_CUDA;
}

// Blocks per plane of the influence kernel: about a thousand in all.
int influence_blocks(int m1, int m2, int m3) {
  const int need = grid_for((long long)m2 * (m3 / 2 + 1), 256);
  return std::min(need, std::max(1, 1024 / m1));
}

// Grid-size dependent state: plan, moduli, grid buffers.
int spme_setup(SpmeWork &c, int n, int m1, int m2, int m3, int nbsp, cudaStream_t s) {
  // planes on the y grid dimension, 32-bit plane and atom indices
  if (m1 > 65535 || (long long)m2 * m3 > (1LL << 30) || n > (1 << 28)) return MDBAS_NB_ERR_ARG;
  int dev = 0;
  MDB_CUDA(cudaGetDevice(&dev));
  const long long mm = (long long)m1 * m2 * m3;
  if (!c.planBackValid || c.m1 != m1 || c.m2 != m2 || c.m3 != m3 || c.device != dev) {
    c.drop_plans();
    MDB_TRY(cufft_check(cufftPlan3d(&c.plan, m1, m2, m3, CUFFT_D2Z), "cufftPlan3d"));
    c.planValid = true;
    MDB_TRY(cufft_check(cufftPlan3d(&c.planBack, m1, m2, m3, CUFFT_Z2D), "cufftPlan3d"));
    c.planBackValid = true;
    c.m1 = m1;
    c.m2 = m2;
    c.m3 = m3;
    c.device = dev;
    c.nbsp = 0;
    c.haloSmem = 0;  // a function attribute is per device
  }
  MDB_TRY(cufft_check(cufftSetStream(c.plan, s), "cufftSetStream"));
  MDB_TRY(cufft_check(cufftSetStream(c.planBack, s), "cufftSetStream"));
  if (c.nbsp != nbsp) {
    std::vector<double> bm(m1 + m2 + m3);
    bsp_moduli(m1, nbsp, bm.data());
    bsp_moduli(m2, nbsp, bm.data() + m1);
    bsp_moduli(m3, nbsp, bm.data() + m1 + m2);
    MDB_TRY(c.bmod.ensure(sizeof(double) * bm.size()));
    MDB_CUDA(cudaMemcpy(c.bmod.p, bm.data(), sizeof(double) * bm.size(), cudaMemcpyHostToDevice));
    c.nbsp = nbsp;
  }
  MDB_TRY(c.qsp.ensure(sizeof(double) * mm));
  MDB_TRY(c.ft.ensure(sizeof(cufftDoubleComplex) * (size_t)m1 * m2 * (m3 / 2 + 1)));
  MDB_TRY(c.spl.ensure(sizeof(double) * 6 * (size_t)nbsp * n));
  MDB_TRY(c.cell.ensure(sizeof(int) * 3 * (size_t)n));
  MDB_TRY(c.fr.ensure(sizeof(double) * 3 * (size_t)n));
  MDB_TRY(c.sums.ensure(sizeof(double) * 16));
  if (!c.done.p) {
    MDB_TRY(c.done.ensure(sizeof(unsigned)));
    MDB_CUDA(cudaMemsetAsync(c.done.p, 0, sizeof(unsigned), s));
  }
  {
    // per-block partial sums: influence (7 x blocks), then forces (3 x blocks)
    const long long gF = ((long long)n * 16 + 255) / 256;
    const long long nt = (long long)(m1 / 8) * (m2 / 8) * (m3 / 8);
    MDB_TRY(c.part.ensure(sizeof(double) * (size_t)std::max(
                              7LL * influence_blocks(m1, m2, m3) * m1, 3 * std::max(gF, nt))));
  }
  {
    const int nt = (m1 / 8) * (m2 / 8) * (m3 / 8);
    MDB_TRY(c.tileOf.ensure(sizeof(int) * (size_t)n));
    MDB_TRY(c.tileList.ensure(sizeof(int) * (size_t)n));
    MDB_TRY(c.tileSorted.ensure(sizeof(int) * (size_t)n));
    MDB_TRY(c.tileCount.ensure(sizeof(int) * (size_t)(nt + 1)));
    MDB_TRY(c.tileStart.ensure(sizeof(int) * (size_t)(nt + 1)));
    MDB_TRY(c.tileFill.ensure(sizeof(int) * (size_t)(nt + 1)));
    if (nt > 0) {
      const int H = kSpTile + nbsp - 1;
      const int smem = (int)sizeof(double) * H * H * H;
      MDB_TRY(c.halo.ensure(sizeof(double) * (size_t)nt * H * H * H));
      if (smem > c.haloSmem) {  // set once, before any capture of these launches
        MDB_CUDA(cudaFuncSetAttribute(k_spme_spread_halo<1>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        MDB_CUDA(cudaFuncSetAttribute(k_spme_spread_halo<kSpPts>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        MDB_CUDA(cudaFuncSetAttribute(k_spme_forces_tiled<0>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        c.haloSmem = smem;
      }
    }
  }
  c.n = n;
  return MDBAS_NB_OK;
}

// The whole computation on device arrays; forces (minus their mean) are added
// to fx/fy/fz; out[0] = reciprocal energy + self + non-neutral, out[1] =
// virial, out[2..7] = stress (MDBas's 6-component layout).
int spme_launch_impl(SpmeWork &c, int n, const PBC *box, double alpha, double chargeConst,
                     int m1, int m2, int m3, int nbsp, const double *x, const double *y,
                     const double *z, const double *q, double *fx, double *fy, double *fz,
                     cudaStream_t s) {
  MDB_TRY(spme_setup(c, n, m1, m2, m3, nbsp, s));
  const SpmeBox b = make_spme_box(box);
  const long long mm = (long long)m1 * m2 * m3;
  double *sums = c.sums.as<double>();  // 0-5 stress, 6 energy, 7-9 force sums
  const bool tiled = m1 % kSpTile == 0 && m2 % kSpTile == 0 && m3 % kSpTile == 0;
  const int nt1 = m1 / kSpTile, nt2 = m2 / kSpTile, nt3 = m3 / kSpTile;
  const int nt = nt1 * nt2 * nt3;
  {
    double *spl = c.spl.as<double>();
    int *cel = c.cell.as<int>();
    int *tof = tiled ? c.tileOf.as<int>() : nullptr, *cnt = c.tileCount.as<int>();
    if (tiled) MDB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)(nt + 1), s));
    const auto kern = nbsp == 8   ? k_spme_splines<8>
                      : nbsp == 6 ? k_spme_splines<6>
                      : nbsp == 4 ? k_spme_splines<4>
                                  : k_spme_splines<0>;
    MDB_LAUNCH(kern, grid_for(3LL * n, kSplThreads), kSplThreads, 0, s, n, b, m1, m2, m3, nbsp, x,
               y, z, spl, cel, tof, cnt);
  }
  if (tiled) {
    // deterministic: bins of atoms per 8^3 tile, one block per tile
    const int reach = 1 + (nbsp + kSpTile - 2) / kSpTile;  // halo boxes covering a point, per dim
    MDB_LAUNCH(k_spme_tile_scan, 1, 1024, 0, s, nt, c.tileCount.as<int>(), c.tileStart.as<int>(),
               c.tileFill.as<int>());
    MDB_LAUNCH(k_spme_tile_fill, grid_for(n, 256), 256, 0, s, n, c.tileOf.as<int>(),
               c.tileStart.as<int>(), c.tileFill.as<int>(), c.tileList.as<int>());
    const bool rows = nbsp == 8 || nbsp == 6 || nbsp == 4;  // these sort their bins themselves
    if (!rows)
      MDB_LAUNCH(k_spme_tile_sort, nt, 64, 0, s, c.tileStart.as<int>(), c.tileList.as<int>(),
                 c.tileSorted.as<int>());
    const int H = kSpTile + nbsp - 1;
    const int *tst = c.tileStart.as<int>();
    const double *spl = c.spl.as<double>();
    const int *cel = c.cell.as<int>();
    double *hal = c.halo.as<double>();
    const int *tli = c.tileList.as<int>();
    int *tso = c.tileSorted.as<int>();
    const auto spread = nbsp == 8   ? k_spme_spread_rows<8>
                        : nbsp == 6 ? k_spme_spread_rows<6>
                                    : k_spme_spread_rows<4>;
    if (rows)
      MDB_LAUNCH(spread, nt, 256, 0, s, nt2, nt3, q, spl, cel, tst, tli, tso, hal);
    else if (nbsp <= 8)
      MDB_LAUNCH(k_spme_spread_halo<1>, nt, 512, sizeof(double) * H * H * H, s, nbsp, nt2, nt3,
                 q, c.spl.as<double>(), c.cell.as<int>(), c.tileStart.as<int>(),
                 c.tileSorted.as<int>(), c.halo.as<double>());
    else
      MDB_LAUNCH(k_spme_spread_halo<kSpPts>, nt, 512, sizeof(double) * H * H * H, s, nbsp, nt2,
                 nt3, q, c.spl.as<double>(), c.cell.as<int>(), c.tileStart.as<int>(),
                 c.tileSorted.as<int>(), c.halo.as<double>());
    const dim3 gg(grid_for((long long)m2 * m3, 256), m1);
    double *qs = c.qsp.as<double>();
    const auto gather = nbsp == 8   ? k_spme_halo_gather2<8>
                        : nbsp == 6 ? k_spme_halo_gather2<6>
                                    : k_spme_halo_gather2<4>;
    if (rows)
      MDB_LAUNCH(gather, gg, 256, 0, s, m2, m3, nt1, nt2, nt3, hal, qs);
    else
      MDB_LAUNCH(k_spme_halo_gather, gg, 256, 0, s, m1, m2, m3, nbsp, reach, nt1, nt2, nt3, hal,
                 qs);
  } else {
    MDB_CUDA(cudaMemsetAsync(c.qsp.p, 0, sizeof(double) * mm, s));
    MDB_LAUNCH(k_spme_spread, grid_for((long long)n * nbsp, 128), 128, 0, s, n, m1, m2, m3,
               nbsp, q, c.spl.as<double>(), c.cell.as<int>(), c.qsp.as<double>());
  }
  // the charge grid forward, its influence-weighted transform back over it
  double *grid = c.qsp.as<double>();
  cufftDoubleComplex *ft = c.ft.as<cufftDoubleComplex>();
  MDB_TRY(cufft_check(cufftExecD2Z(c.plan, grid, ft), "cufftExecD2Z"));
  const double rvol = 6.283185307179586 / b.vol;
  const double ralpha2 = -0.25 / (alpha * alpha);
  double rc = fmin((double)m1 * b.u, (double)m2 * b.v);
  rc = fmin(rc, (double)m3 * b.w) * 1.05 * 6.283185307179586;
  double *part = c.part.as<double>();
  unsigned *done = c.done.as<unsigned>();
  MDB_LAUNCH(k_spme_influence, dim3(influence_blocks(m1, m2, m3), m1), 256, 0, s, m1, m2, m3, b,
             ralpha2, rc * rc, c.bmod.as<double>(), ft, part, done, sums);
  MDB_TRY(cufft_check(cufftExecZ2D(c.planBack, ft, grid), "cufftExecZ2D"));
  int group = 1;
  while (group < nbsp) group <<= 1;
  if (tiled) {
    const int H = kSpTile + nbsp - 1;
    const size_t smem = sizeof(double) * H * H * H;
    const double f2 = -2.0 * rvol * chargeConst;
    const int *tst = c.tileStart.as<int>(), *tso = c.tileSorted.as<int>();
    const double *spl = c.spl.as<double>();
    const int *cel = c.cell.as<int>();
    double *frr = c.fr.as<double>();
    const auto kern = nbsp == 8   ? k_spme_forces_tiled<8>
                      : nbsp == 6 ? k_spme_forces_tiled<6>
                      : nbsp == 4 ? k_spme_forces_tiled<4>
                                  : k_spme_forces_tiled<0>;
    MDB_LAUNCH(kern, nt, 256, smem, s, n, m1, m2, m3, nbsp, group, nt2, nt3, b, f2, q, spl, cel,
               tst, tso, grid, frr, part, done, sums + 7);
  } else {
    MDB_LAUNCH(k_spme_forces, grid_for((long long)n * group, 256), 256, 0, s, n, m1, m2, m3, nbsp,
               group, b, -2.0 * rvol * chargeConst, q, c.spl.as<double>(), c.cell.as<int>(), grid,
               c.fr.as<double>(), part, done, sums + 7);
  }
  c.f1 = rvol * chargeConst;
  return fx ? spme_add(c, n, fx, fy, fz, s) : MDBAS_NB_OK;
}

// Energy, virial and stress from the device sums h (src/spme.c:577-640).
void spme_results(const PBC *box, double alpha, double chargeConst, double systq, double sumq2,
                  const double *h, double out[8]) {
  const double rvol = 6.283185307179586 / box->vol;
  const double eself = -chargeConst * alpha * sumq2 / kSqrtPi;
  const double enn = -(0.5 * 3.141592653589793 * chargeConst) *
                     ((systq / alpha) * (systq / alpha) / box->vol);
  const double fact1 = rvol * chargeConst;
  const double erec = h[kSpmeEnergy];
  double st[6];
  st[0] = fact1 * (h[0] + erec) + enn;
  st[1] = fact1 * h[1];
  st[2] = fact1 * h[2];
  st[3] = fact1 * (h[3] + erec) + enn;
  st[4] = fact1 * h[4];
  st[5] = fact1 * (h[5] + erec) + enn;
  out[0] = fact1 * erec + eself + enn;
  out[1] = -(st[0] + st[3] + st[5]);
  for (int k = 0; k < 6; ++k) out[2 + k] = st[k];
}

int spme_run(int n, const PBC *box, double alpha, double chargeConst, int m1, int m2, int m3,
             int nbsp, const double *x, const double *y, const double *z, const double *q,
             double systq, double sumq2, double *fx, double *fy, double *fz, double out[8],
             cudaStream_t s) {
  SpmeWork &c = spme_ctx();
  MDB_TRY(spme_launch_impl(c, n, box, alpha, chargeConst, m1, m2, m3, nbsp, x, y, z, q, fx, fy,
                           fz, s));
  double h[16];
  MDB_CUDA(cudaMemcpyAsync(h, c.sums.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  MDB_CUDA(cudaStreamSynchronize(s));
  spme_results(box, alpha, chargeConst, systq, sumq2, h, out);
  return MDBAS_NB_OK;
}

int check_grid(int m1, int m2, int m3, int nbsp) {
  if (m1 <= 0 || m2 <= 0 || m3 <= 0 || nbsp < 2 || nbsp > kMaxOrder) return MDBAS_NB_ERR_ARG;
  if (nbsp > m1 || nbsp > m2 || nbsp > m3) return MDBAS_NB_ERR_ARG;
  return MDBAS_NB_OK;
}

int nint_h(double x) { return (x >= 0.) ? (int)(x + 0.5) : (int)(x - 0.5); }

}  // namespace

int mdbas::spme_add(SpmeWork &c, int n, double *fx, double *fy, double *fz, cudaStream_t s) {
  MDB_LAUNCH(k_spme_add, grid_for(n, 256), 256, 0, s, n, c.fr.as<double>(),
             c.sums.as<double>() + 7, fx, fy, fz);
  return MDBAS_NB_OK;
}

int mdbas::spme_launch(SpmeWork &c, int n, const PBC *box, double alpha, double chargeConst,
                       int m1, int m2, int m3, int nbsp, const double *x, const double *y,
                       const double *z, const double *q, double *fx, double *fy, double *fz,
                       cudaStream_t s) {
  return spme_launch_impl(c, n, box, alpha, chargeConst, m1, m2, m3, nbsp, x, y, z, q, fx, fy, fz,
                          s);
}

extern "C" {

int mdbas_nb_spme(int nAtom, const PBC *box, double alpha, double chargeConst, int m1, int m2,
                  int m3, int nbsp, const double *x, const double *y, const double *z,
                  const double *q, double *fx, double *fy, double *fz, double out[8],
                  int device_ptrs, void *stream) {
  if (nAtom <= 0 || !box || !x || !y || !z || !q || !fx || !fy || !fz || !out || !(alpha > 0.))
    return MDBAS_NB_ERR_ARG;
  MDB_TRY(check_grid(m1, m2, m3, nbsp));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  SpmeWork &c = spme_ctx();
  double systq = 0., sumq2 = 0.;
  std::vector<double> hq;
  const double *qh = q;
  if (device_ptrs) {
    hq.resize(nAtom);
    MDB_CUDA(cudaMemcpy(hq.data(), q, sizeof(double) * nAtom, cudaMemcpyDeviceToHost));
    qh = hq.data();
  }
  charge_sums(nAtom, qh, &systq, &sumq2);
  if (device_ptrs)
    return spme_run(nAtom, box, alpha, chargeConst, m1, m2, m3, nbsp, x, y, z, q, systq, sumq2,
                    fx, fy, fz, out, s);
  // host arrays: stage through device buffers; forces are added to the
  // caller's arrays
  standalone_copies();
  MDB_TRY(c.xyzq.ensure(sizeof(double) * 4 * (size_t)nAtom));
  MDB_TRY(c.fout.ensure(sizeof(double) * 3 * (size_t)nAtom));
  double *d = c.xyzq.as<double>(), *f = c.fout.as<double>();
  const size_t bytes = sizeof(double) * (size_t)nAtom;
  const CopySpan in[4] = {
      {const_cast<double *>(x), d, bytes},
      {const_cast<double *>(y), d + nAtom, bytes, false, true},
      {const_cast<double *>(z), d + 2 * (size_t)nAtom, bytes, false, true},
      {const_cast<double *>(q), d + 3 * (size_t)nAtom, bytes, false, true}};
  MDB_TRY(copy_in(in, 4, s));
  MDB_CUDA(cudaMemsetAsync(f, 0, 3 * bytes, s));
  double h[16];
  MDB_TRY(spme_launch_impl(c, nAtom, box, alpha, chargeConst, m1, m2, m3, nbsp, d, d + nAtom,
                           d + 2 * (size_t)nAtom, d + 3 * (size_t)nAtom, f, f + nAtom,
                           f + 2 * (size_t)nAtom, s));
  const CopySpan3 f3(fx, fy, fz, f, nAtom, true);
  const CopySpan o[4] = {f3.s[0], f3.s[1], f3.s[2], {h, c.sums.p, sizeof(h)}};
  MDB_TRY(copy_out(o, 4, s));
  spme_results(box, alpha, chargeConst, systq, sumq2, h, out);
  return MDBAS_NB_OK;
}

// MDBas's init_spme (src/spme.c:32-68): the grid of the reciprocal sum.
void init_spme(CTRL *ctrl, PARAM *param, EWALD *ewald, PBC *box) {
  ewald->prec = fmin(fabs(ewald->prec), 0.5);
  ewald->tol = sqrt(fabs(log(ewald->prec * param->cutOff)));
  if (!ctrl->keyAlpha)
    ewald->alpha = sqrt(fabs(log(ewald->prec * param->cutOff * ewald->tol))) / param->cutOff;
  const double ta = 2.0 * ewald->tol * ewald->alpha;
  ewald->tol1 = sqrt(-log(ewald->prec * param->cutOff * (ta * ta)));
  if (!ctrl->keyMmax) {
    ewald->m1max = nint_h(0.25 + box->pa * ewald->alpha * ewald->tol1 / 3.141592653589793);
    ewald->m2max = nint_h(0.25 + box->pb * ewald->alpha * ewald->tol1 / 3.141592653589793);
    ewald->m3max = nint_h(0.25 + box->pc * ewald->alpha * ewald->tol1 / 3.141592653589793);
  }
  int *m[3] = {&ewald->m1max, &ewald->m2max, &ewald->m3max};
  for (int d = 0; d < 3; ++d) {
    int p2 = 1;
    while (*m[d] > p2 && p2 < 256) p2 *= 2;
    *m[d] = 2 * p2;
  }
  ewald->mmax = ewald->m1max * ewald->m2max * ewald->m3max;
}

void spme_free(PARAM *param) { (void)param; }

// MDBas's spme_energy (src/spme.c:357-700) on the GPU.  As in MDBas the
// mean over the whole force arrays is removed after the reciprocal forces
// are added (energy() calls it first, on zeroed arrays).
double spme_energy(PARAM *param, EWALD *ewald, PBC *box, const double x[], const double y[],
                   const double z[], double fx[], double fy[], double fz[], const double q[],
                   double stress[6], double *virEwaldRec) {
  const int n = param->nAtom;
  std::vector<double> rx(n, 0.), ry(n, 0.), rz(n, 0.);
  double out[8];
  const int st = mdbas_nb_spme(n, box, ewald->alpha, param->chargeConst, ewald->m1max,
                               ewald->m2max, ewald->m3max, ewald->nbsp, x, y, z, q, rx.data(),
                               ry.data(), rz.data(), out, 0, nullptr);
  if (st != MDBAS_NB_OK) {
    fprintf(stderr, "spme_energy (GPU): %s: %s\n", mdbas_nb_status_string(st),
            mdbas_nb_last_message());
    exit(1);
  }
  double mx = 0., my = 0., mz = 0.;
  for (int i = 0; i < n; ++i) {
    fx[i] += rx[i];
    fy[i] += ry[i];
    fz[i] += rz[i];
    mx += fx[i];
    my += fy[i];
    mz += fz[i];
  }
  // rx had its own mean removed; MDBas removes the mean of the whole array
  mx /= (double)n;
  my /= (double)n;
  mz /= (double)n;
  for (int i = 0; i < n; ++i) {
    fx[i] -= mx;
    fy[i] -= my;
    fz[i] -= mz;
  }
  for (int k = 0; k < 6; ++k) stress[k] = out[2 + k];
  *virEwaldRec = out[1];
  return out[0];
}

}  // extern "C"
