// list_ref.cu -- MDBas-format half Verlet lists built on the GPU.
//
// Two builders with MDBas's exact output (same entries in the same order):
//
//  * link cells (link_cell_verlet_list[_update], src/list.c:1793-2619): atoms
//    are binned with MDBas's FP64 fractional coordinates; each cell lists its
//    atoms in descending index (MDBas's LIFO head/link chains); neighOrder is
//    that cell-major order; atom i scans the stencil cells in table order
//    (link_stencil.h) and, in its own cell, only the atoms after it.
//  * all pairs (verlet_list[_update], src/list.c:896-1123): j = i+1..N-1 with
//    MDBas's dist() minimum image; neighOrder is the identity.
//
// Layout: after binning, positions/fractional coordinates are gathered into
// cell order so that a warp scanning a cell reads consecutive addresses.  Each
// candidate pair is tested once: one warp takes eight atoms i and 32
// consecutive candidates at a time, the test's ballot is the word of a bit
// mask (atom, candidate), a second kernel clears the excluded pairs and
// counts the bits, and after the scan of the counts in neighOrder order a
// third writes the entries in bit order, which is the order MDBas's serial
// loop visits them in.
//
// The test itself runs in FP32 on box coordinates; a pair whose FP32 r^2 lies
// within the rounding bound of (rc+delr)^2 is settled by MDBas's FP64
// expression, so the list is MDBas's, entry by entry.  A build of the
// 96,000-atom box takes 0.62 ms (tests 0.31, counts 0.05, entries 0.17); FP64
// tests, once to count and once to fill, took 2.50.  All pairs of 3,000 atoms:
// 0.134 -> 0.072 ms.
//
// The FP64 arithmetic uses __dadd_rn/__dmul_rn (no FMA contraction) in
// MDBas's association order, so every r^2 <= (rc+delr)^2 decision is the
// one MDBas's x86 build makes.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "link_stencil.h"
#include "list_ref.cuh"

namespace mdbas {

namespace {

constexpr int kMaxRatio = 5;
constexpr int kInvSide = 2 * kMaxRatio + 1;
__constant__ int c_stencil[LINK_STENCIL_MAX * 3];
// stencil entry of a cell offset (-5..5 per axis), -1 where there is none
__constant__ short c_stencilOf[kInvSide * kInvSide * kInvSide];

constexpr int kGroup = 8;       // atoms i per warp of the candidate tests
constexpr int kListWarps = 4;   // warps per block of the list kernels
constexpr int kPiece = 32;      // candidate chunks per warp of the tests
constexpr int kTestWarps = 4096;  // of the tests before groups of atoms are split

// image_update (src/utils.c:162-218), in place.
__global__ void k_image_update(int n, DevBox b, double *x, double *y, double *z) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double xi = x[i], yi = y[i], zi = z[i];
  image_d(b, xi, yi, zi);
  x[i] = xi;
  y[i] = yi;
  z[i] = zi;
}

// Fractional coordinates + 0.5 (src/list.c:1932-1937) and the link cell
// (src/list.c:1943-1955): truncation toward zero, clamped above only.
__global__ void k_lc_bin(int n, DevBox b, int nlcx, int nlcy, int nlcz,
                         const double *__restrict__ x, const double *__restrict__ y,
                         const double *__restrict__ z, double *__restrict__ xu,
                         double *__restrict__ yu, double *__restrict__ zu,
                         int *__restrict__ cellOf, int *__restrict__ cellCount,
                         int *__restrict__ flags) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double xi = x[i], yi = y[i], zi = z[i];
  const double a = dadd(dadd(dadd(dmul(xi, b.u1), dmul(yi, b.u2)), dmul(zi, b.u3)), 0.5);
  const double c = dadd(dadd(dadd(dmul(xi, b.v1), dmul(yi, b.v2)), dmul(zi, b.v3)), 0.5);
  const double d = dadd(dadd(dadd(dmul(xi, b.w1), dmul(yi, b.w2)), dmul(zi, b.w3)), 0.5);
  xu[i] = a;
  yu[i] = c;
  zu[i] = d;
  if (!(isfinite(a) && isfinite(c) && isfinite(d))) {
    atomicOr(flags, FLAG_NONFINITE);
    cellOf[i] = -1;
    return;
  }
  int ix = __double2int_rz(dmul((double)nlcx, a));
  int iy = __double2int_rz(dmul((double)nlcy, c));
  int iz = __double2int_rz(dmul((double)nlcz, d));
  ix = min(ix, nlcx - 1);
  iy = min(iy, nlcy - 1);
  iz = min(iz, nlcz - 1);
  if (ix < 0 || iy < 0 || iz < 0) {
    // MDBas would index head[] out of bounds here; report instead.
    atomicOr(flags, FLAG_OUTSIDE);
    cellOf[i] = -1;
    return;
  }
  const int cell = ix + nlcx * (iy + nlcy * iz);
  cellOf[i] = cell;
  atomicAdd(cellCount + cell, 1);
}

__global__ void k_lc_scatter(int n, const int *__restrict__ cellOf,
                             const int *__restrict__ cellStart, int *__restrict__ cellFill,
                             int *__restrict__ tmpIdx) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cellOf[i];
  if (c < 0) return;
  const int slot = atomicAdd(cellFill + c, 1);
  tmpIdx[cellStart[c] + slot] = i;
}

// Order each cell's atoms by descending index (MDBas's LIFO chain order):
// the rank of a member is the number of members with a larger index.
__global__ void k_lc_order(int ncell, const int *__restrict__ cellStart,
                           const int *__restrict__ tmpIdx, int *__restrict__ sortedIdx) {
  __shared__ int chunk[1024];
  const int c = blockIdx.x;
  if (c >= ncell) return;
  const int s = cellStart[c], e = cellStart[c + 1];
  for (int base = s; base < e; base += blockDim.x) {
    const int m = base + threadIdx.x;
    const int mine = (m < e) ? tmpIdx[m] : -1;
    int rank = 0;
    for (int cb = s; cb < e; cb += 1024) {
      const int cnt = min(1024, e - cb);
      __syncthreads();
      for (int t = threadIdx.x; t < cnt; t += blockDim.x) chunk[t] = tmpIdx[cb + t];
      __syncthreads();
      if (m < e)
        for (int t = 0; t < cnt; ++t) rank += (chunk[t] > mine);
    }
    if (m < e) sortedIdx[s + rank] = mine;
  }
}

// Cell order: fractional coordinates for the exact test, FP32 box coordinates
// (x, y, z, frozen) for the first one.  An atom more than two box lengths
// from the origin gets NaN there: its pairs go to the exact test.
__global__ void k_lc_gather(int ncell, DevBox b, const int *__restrict__ cellStart,
                            const int *__restrict__ sortedIdx, const double *__restrict__ xu,
                            const double *__restrict__ yu, const double *__restrict__ zu,
                            const int *__restrict__ frozen, double *__restrict__ xs,
                            double *__restrict__ ys, double *__restrict__ zs,
                            float4 *__restrict__ cs, int *__restrict__ posOf) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= cellStart[ncell]) return;
  const int i = sortedIdx[p];
  const double u = xu[i], v = yu[i], w = zu[i];
  xs[p] = u;
  ys[p] = v;
  zs[p] = w;
  float4 c;
  c.x = (float)(u * b.a1 + v * b.b1 + w * b.c1);
  c.y = (float)(u * b.a2 + v * b.b2 + w * b.c2);
  c.z = (float)(u * b.a3 + v * b.b3 + w * b.c3);
  if (!(fabs(u) <= 2. && fabs(v) <= 2. && fabs(w) <= 2.)) c.x = __int_as_float(0x7fc00000);
  c.w = frozen && frozen[i] ? 1.f : 0.f;
  cs[p] = c;
  posOf[i] = p;
}

// Neighbour cell l of cell (ix, iy, iz) and its periodic image (in boxes).
__device__ __forceinline__ int stencil_cell(int l, int ix, int iy, int iz, int nx, int ny, int nz,
                                            int &sx, int &sy, int &sz) {
  int jx = ix + c_stencil[3 * l], jy = iy + c_stencil[3 * l + 1], jz = iz + c_stencil[3 * l + 2];
  sx = sy = sz = 0;
  if (jx > nx - 1) { jx -= nx; sx = 1; } else if (jx < 0) { jx += nx; sx = -1; }
  if (jy > ny - 1) { jy -= ny; sy = 1; } else if (jy < 0) { jy += ny; sy = -1; }
  if (jz > nz - 1) { jz -= nz; sz = 1; } else if (jz < 0) { jz += nz; sz = -1; }
  return jx + nx * (jy + ny * jz);
}

// A cell's row in the candidate tables: its number, or, where there are more
// cells than atoms (byStart), the position of its first atom, which no other
// occupied cell has.  So the tables have min(cells, atoms) rows: a droplet of
// 3,000 atoms in a 2,000 A box has 2.9 million cells.
__device__ __forceinline__ size_t table_row(int byStart, int cell, const int *cellStart) {
  return byStart ? cellStart[cell] : cell;
}

// Candidate chunks of every occupied cell, one warp per cell (byStart: per
// atom, of which the first of its cell goes on): chunkOff[l], the first chunk of
// stencil cell l (its atoms in runs of 32), chunkOff[cellCheck] the total, and
// chunkBase[c], the first position of chunk c.  A total beyond stride raises
// FLAG_CELL and goes to *need.
__global__ void __launch_bounds__(32 * kListWarps)
k_lc_chunks(int ncell, int nx, int ny, int nz, int cellCheck, int stride, int byStart,
            const int *__restrict__ cellStart, const int *__restrict__ cellOf,
            const int *__restrict__ order, int *__restrict__ chunkOff,
            int *__restrict__ chunkBase, int *__restrict__ flags, int *__restrict__ need) {
  const int lane = threadIdx.x & 31;
  int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (byStart) {
    const int p = k;
    if (p >= cellStart[ncell]) return;
    k = cellOf[order[p]];
    if (cellStart[k] != p) return;
  } else if (k >= ncell || cellStart[k] == cellStart[k + 1]) {
    return;
  }
  const int ix = k % nx, iy = (k / nx) % ny, iz = k / (nx * ny);
  const size_t row = table_row(byStart, k, cellStart);
  int *off = chunkOff + row * (cellCheck + 1);
  int *base = chunkBase + row * stride;
  int run = 0;
  for (int l0 = 0; l0 < cellCheck; l0 += 32) {
    const int l = l0 + lane;
    int lo = 0, nc = 0;
    if (l < cellCheck) {
      int sx, sy, sz;
      const int ll = stencil_cell(l, ix, iy, iz, nx, ny, nz, sx, sy, sz);
      lo = cellStart[ll];
      nc = (cellStart[ll + 1] - lo + 31) >> 5;
    }
    int x = nc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (l < cellCheck) {
      const int first = run + x - nc;
      off[l] = first;
      for (int c = 0; c < nc && first + c < stride; ++c) base[first + c] = lo + 32 * c;
    }
    run += __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) {
    off[cellCheck] = run;
    if (run > stride) {
      atomicOr(flags, FLAG_CELL);
      atomicMax(need, run);
    }
  }
}

// Where the candidates of atom p lie: chunks [first, last) of its mask row.
// Link cells: atoms are tested in runs, the part of a group of `group` (at
// most kGroup) consecutive positions that lies in one cell; chunks of the own cell before
// the run hold no candidate.  All pairs: chunk c is atoms 32c .. 32c + 31.
struct ChunkMap {
  int linkCells, n, stride, cellCheck, ncell, byStart, group, nlc[3];
  const int *cellStart, *cellOf, *order, *posOf, *chunkOff, *chunkBase;

  __device__ __forceinline__ int atoms() const { return linkCells ? cellStart[ncell] : n; }
  __device__ __forceinline__ int atom(int p) const { return linkCells ? order[p] : p; }
  __device__ __forceinline__ const int *offsets(int cell) const {
    return chunkOff + table_row(byStart, cell, cellStart) * (cellCheck + 1);
  }
  __device__ __forceinline__ void range(int p, int cell, int &first, int &last) const {
    const int g0 = p & ~(group - 1);
    if (linkCells) {
      const int s = cellStart[cell];
      first = (max(g0, s) + 1 - s) >> 5;
      last = offsets(cell)[cellCheck];
    } else {
      first = (g0 + 1) >> 5;
      last = (n + 31) >> 5;
    }
  }
};

// The row words of up to kGroup atoms, kept one per lane until four chunks
// are done: lane 4 g + c holds word c of atom g, so a store writes 16 bytes
// of every row.
struct RowWords {
  unsigned word = 0;
  __device__ __forceinline__ void put(int lane, int g, int c, unsigned m) {
    if (lane == 4 * g + (c & 3)) word = m;
  }
  // All atoms' words of chunk c: lane 4 g + c takes atom g's by halving.
  __device__ __forceinline__ void put_all(int lane, int c, const unsigned (&m)[kGroup]) {
    const bool g0 = lane & 4, g1 = lane & 8, g2 = lane & 16;
    const unsigned a0 = g0 ? m[1] : m[0], a1 = g0 ? m[3] : m[2];
    const unsigned a2 = g0 ? m[5] : m[4], a3 = g0 ? m[7] : m[6];
    const unsigned b0 = g1 ? a1 : a0, b1 = g1 ? a3 : a2;
    if ((lane & 3) == (c & 3)) word = g2 ? b1 : b0;
  }
  __device__ __forceinline__ void flush(int lane, int c, int atoms, unsigned *rows, int stride) {
    const int g = lane >> 2;
    if (g < atoms) rows[(size_t)g * stride + (c & ~3) + (lane & 3)] = word;
    word = 0;
  }
};

// Bits of a chunk starting at `base` that come after position p.
__device__ __forceinline__ unsigned bits_after(int p, int base) {
  const int s = p - base;
  return s < 0 ? 0xffffffffu : s >= 31 ? 0u : 0xffffffffu << (s + 1);
}

// Candidate tests, link cells: one warp per group of map.group positions in
// [p0, p1) (p0 a multiple of kGroup) and piece of kPiece chunks (grid y); rows
// of masks start at p0.
// rl2 = (rc+delr)^2; band bounds the error of the FP32 r^2 near rl2.
// Bound by instruction issue: per candidate word 6 FP32 operations, two
// compares and a ballot, the candidate's load shared by the group.  (Boxes
// around the chunks, to skip those out of reach, took away a fifth of the
// tests' instructions and gave it back in the boxes' own kernels.)
template <bool FROZEN>
__global__ void __launch_bounds__(32 * kListWarps)
k_lc_masks(int p0, int p1, DevBox b, ChunkMap map, double cutnb2, float rl2, float band,
           const double *__restrict__ xs, const double *__restrict__ ys,
           const double *__restrict__ zs, const float4 *__restrict__ cs,
           const int *__restrict__ flags, unsigned *__restrict__ masks) {
  const int lane = threadIdx.x & 31;
  const int g0 = p0 + map.group * (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int end = min(min(g0 + map.group, p1), map.atoms());
  if (g0 >= end || (*flags & FLAG_CELL)) return;
  const int nx = map.nlc[0], ny = map.nlc[1], nz = map.nlc[2];
  for (int p = g0; p < end;) {
    const int k = map.cellOf[map.order[p]];
    const int ix = k % nx, iy = (k / nx) % ny, iz = k / (nx * ny);
    const int atoms = min(map.cellStart[k + 1], end) - p;
    float x[kGroup], y[kGroup], z[kGroup];
    unsigned frozenRows = 0;
#pragma unroll
    for (int g = 0; g < kGroup; ++g) {
      // rows that are not there: far from everything
      x[g] = 1e18f;
      y[g] = z[g] = 0.f;
      if (g < atoms) {
        const float4 c = cs[p + g];
        x[g] = c.x;
        y[g] = c.y;
        z[g] = c.z;
        if (FROZEN && c.w != 0.f) frozenRows |= 1u << g;
      }
    }
    unsigned *rows = masks + (size_t)(p - p0) * map.stride;
    // this warp's piece of the chunks, from the first that holds a position
    // after p
    const int *off = map.offsets(k);
    const int cFirst = max((p + 1 - map.cellStart[k]) >> 5, (int)blockIdx.y * kPiece);
    const int cLast = min(off[map.cellCheck], (int)(blockIdx.y + 1) * kPiece);
    if (cFirst >= cLast) {
      p += atoms;
      continue;
    }
    RowWords words;
    int c = cFirst;
    // the chunks of stencil cell l; OWN: the cell itself, where only
    // positions after atom p + g count
    const auto scan = [&](int l, auto own) {
      constexpr bool OWN = decltype(own)::value;
      int sx, sy, sz;
      const int ll = stencil_cell(l, ix, iy, iz, nx, ny, nz, sx, sy, sz);
      const float ox = (float)(sx * b.a1 + sy * b.b1 + sz * b.c1);
      const float oy = (float)(sx * b.a2 + sy * b.b2 + sz * b.c2);
      const float oz = (float)(sx * b.a3 + sy * b.b3 + sz * b.c3);
      const int hi = map.cellStart[ll + 1];
      int base = map.cellStart[ll] + 32 * (c - off[l]);
      for (; base < hi && c < cLast; base += 32, ++c) {
        const int q = base + lane;
        float4 d = make_float4(-1e18f, 0.f, 0.f, 0.f);
        if (q < hi) d = cs[q];
        d.x += ox;
        d.y += oy;
        d.z += oz;
        bool unsure = false;
        // atoms i that make a pair of two frozen atoms with this candidate
        const unsigned skip = FROZEN && d.w != 0.f ? frozenRows : 0u;
        unsigned m[kGroup];
#pragma unroll
        for (int g = 0; g < kGroup; ++g) {
          const float dx = d.x - x[g], dy = d.y - y[g], dz = d.z - z[g];
          const float t = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, -rl2)));
          unsure |= !(fabsf(t) > band);
          m[g] = __ballot_sync(0xffffffffu, t <= 0.f && !(FROZEN && (skip >> g & 1u)));
          if (OWN) m[g] &= bits_after(p + g, base);
        }
        words.put_all(lane, c, m);
        if (__any_sync(0xffffffffu, unsure)) {
          double xq = 0., yq = 0., zq = 0.;
          if (q < hi) {
            xq = xs[q];
            yq = ys[q];
            zq = zs[q];
          }
          for (int g = 0; g < atoms; ++g) {
            const float4 ci = cs[p + g];
            const float dx = d.x - ci.x, dy = d.y - ci.y, dz = d.z - ci.z;
            const float t = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, -rl2)));
            bool pass = q < hi && t <= 0.f;
            if (q < hi && !(fabsf(t) > band)) {
              const double xt = dadd(dsub(xq, xs[p + g]), (double)sx);
              const double yt = dadd(dsub(yq, ys[p + g]), (double)sy);
              const double zt = dadd(dsub(zq, zs[p + g]), (double)sz);
              const double xd = dadd(dadd(dmul(xt, b.a1), dmul(yt, b.b1)), dmul(zt, b.c1));
              const double yd = dadd(dadd(dmul(xt, b.a2), dmul(yt, b.b2)), dmul(zt, b.c2));
              const double zd = dadd(dadd(dmul(xt, b.a3), dmul(yt, b.b3)), dmul(zt, b.c3));
              pass = dadd(dadd(dmul(xd, xd), dmul(yd, yd)), dmul(zd, zd)) <= cutnb2;
            }
            if (FROZEN && (skip >> g & 1u)) pass = false;
            unsigned m = __ballot_sync(0xffffffffu, pass);
            if (OWN) m &= bits_after(p + g, base);
            words.put(lane, g, c, m);
          }
        }
        if ((c & 3) == 3) words.flush(lane, c, atoms, rows, map.stride);
      }
    };
    // the stencil cell that chunk c lies in, 32 at a time from cell l on (one
    // after the other they are latency: 20,000 atoms spread over 300 A at link
    // ratio 3, of whose 156 stencil cells 11 hold atoms, 673 -> 442 us; 96,000
    // atoms of water at ratio 5 11.1 -> 7.4 ms, at ratio 1 no change)
    const auto holding = [&](int l) {
      for (; l < map.cellCheck; l += 32) {
        const int k = l + lane;
        const unsigned m =
            __ballot_sync(0xffffffffu, k < map.cellCheck && off[k + 1] > c);
        if (m) return l + __ffs(m) - 1;
      }
      return l;
    };
    int l = holding(0);
    if (l == 0) {
      scan(0, std::true_type{});
      l = 1;
    }
    for (; l < map.cellCheck && c < cLast; ++l) {
      if (off[l + 1] <= c) l = holding(l + 1);
      if (l < map.cellCheck) scan(l, std::false_type{});
    }
    if (c & 3) words.flush(lane, c, atoms, rows, map.stride);
    p += atoms;
  }
}

// FP32 coordinates of the all-pairs tests: the atom wrapped into the box
// (NaN, so the exact test, when it lies absurdly far out), and frozen.
__global__ void k_vl_coords(int n, double lx, double ly, double lz, const double *__restrict__ x,
                            const double *__restrict__ y, const double *__restrict__ z,
                            const int *__restrict__ frozen, float4 *__restrict__ cs,
                            int *__restrict__ order) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double xi = x[i], yi = y[i], zi = z[i];
  float4 c;
  c.x = (float)(xi - lx * rint(xi / lx));
  c.y = (float)(yi - ly * rint(yi / ly));
  c.z = (float)(zi - lz * rint(zi / lz));
  if (!(fabs(xi) <= 1e6 * lx && fabs(yi) <= 1e6 * ly && fabs(zi) <= 1e6 * lz))
    c.x = __int_as_float(0x7fc00000);
  c.w = frozen && frozen[i] ? 1.f : 0.f;
  cs[i] = c;
  order[i] = i;
}

// Candidate tests, all pairs: one warp per group of kGroup atoms and piece of
// kPiece chunks (grid y), candidates j > i in index order.  The FP32
// distance takes per axis the smaller of |d| and L - |d| (both atoms in the
// box), two atoms i side by side in packed arithmetic (one by one, the build
// of 12,000 atoms took 171 us, now 148; the link-cell tests, with more loads
// and registers, gained nothing from it); exactOnly: boxes without that form
// take dist() for every pair.
template <bool FROZEN>
__global__ void __launch_bounds__(32 * kListWarps)
k_vl_masks(int p0, int p1, DevBox b, ChunkMap map, double cutnb2, float rl2, float band, float lx,
           float ly, float lz, int exactOnly, const double *__restrict__ xd,
           const double *__restrict__ yd, const double *__restrict__ zd,
           const float4 *__restrict__ cs, unsigned *__restrict__ masks) {
  const int lane = threadIdx.x & 31;
  const int p = p0 + kGroup * (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int n = map.n, atoms = min(p + kGroup, p1) - p;
  if (atoms <= 0) return;
  const int cEnd = min((int)(blockIdx.y + 1) * kPiece, (n + 31) >> 5);
  const int cFirst = max((p + 1) >> 5, (int)blockIdx.y * kPiece);
  if (cFirst >= cEnd) return;
  float2 x[kGroup / 2], y[kGroup / 2], z[kGroup / 2];  // two atoms each, negated
  unsigned frozenRows = 0;
#pragma unroll
  for (int g = 0; g < kGroup; ++g) {
    const float4 c = cs[min(p + g, n - 1)];
    (g & 1 ? x[g / 2].y : x[g / 2].x) = -c.x;
    (g & 1 ? y[g / 2].y : y[g / 2].x) = -c.y;
    (g & 1 ? z[g / 2].y : z[g / 2].x) = -c.z;
    if (FROZEN && c.w != 0.f) frozenRows |= 1u << g;
  }
  // the shorter way round
  const auto image = [](float d, float l) { return fminf(fabsf(d), l - fabsf(d)); };
  unsigned *rows = masks + (size_t)(p - p0) * map.stride;
  RowWords words;
  int c = cFirst;
  for (; c < cEnd; ++c) {
    const int base = 32 * c, q = base + lane;
    const float4 d = cs[min(q, n - 1)];
    bool unsure = exactOnly != 0;
    const unsigned skip = FROZEN && d.w != 0.f ? frozenRows : 0u;
    const unsigned there = n - base >= 32 ? 0xffffffffu : (1u << (n - base)) - 1u;
    unsigned m[kGroup];
#pragma unroll
    for (int g = 0; g < kGroup; g += 2) {
      float2 dx = __fadd2_rn(make_float2(d.x, d.x), x[g / 2]);
      float2 dy = __fadd2_rn(make_float2(d.y, d.y), y[g / 2]);
      float2 dz = __fadd2_rn(make_float2(d.z, d.z), z[g / 2]);
      dx = make_float2(image(dx.x, lx), image(dx.y, lx));
      dy = make_float2(image(dy.x, ly), image(dy.y, ly));
      dz = make_float2(image(dz.x, lz), image(dz.y, lz));
      const float2 t = __ffma2_rn(
          dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, make_float2(-rl2, -rl2))));
      unsure |= !(fabsf(t.x) > band) | !(fabsf(t.y) > band);
      m[g] = __ballot_sync(0xffffffffu, t.x <= 0.f && !(FROZEN && (skip >> g & 1u))) & there;
      m[g + 1] = __ballot_sync(0xffffffffu, t.y <= 0.f && !(FROZEN && (skip >> g & 2u))) & there;
    }
    if (base < p + kGroup)  // the chunks that hold the group itself
#pragma unroll
      for (int g = 0; g < kGroup; ++g) m[g] &= bits_after(p + g, base);
    words.put_all(lane, c, m);
    if (__any_sync(0xffffffffu, unsure)) {
      double xq = 0., yq = 0., zq = 0.;
      if (q < n) {
        xq = xd[q];
        yq = yd[q];
        zq = zd[q];
      }
      for (int g = 0; g < atoms; ++g) {
        const float4 ci = cs[p + g];
        float dx = fabsf(d.x - ci.x), dy = fabsf(d.y - ci.y), dz = fabsf(d.z - ci.z);
        dx = fminf(dx, lx - dx);
        dy = fminf(dy, ly - dy);
        dz = fminf(dz, lz - dz);
        const float t = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, -rl2)));
        bool pass = t <= 0.f;
        if (q < n && (exactOnly || !(fabsf(t) > band))) {
          double ex = dsub(xq, xd[p + g]), ey = dsub(yq, yd[p + g]), ez = dsub(zq, zd[p + g]);
          pass = dist_d(b, ex, ey, ez) <= cutnb2;
        }
        if (FROZEN && (skip >> g & 1u)) pass = false;
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        words.put(lane, g, c, m & there & bits_after(p + g, base));
      }
    }
    if ((c & 3) == 3) words.flush(lane, c, atoms, rows, map.stride);
  }
  if (c & 3) words.flush(lane, c, atoms, rows, map.stride);
}

// One warp per atom of [p0, p1): the pairs that the atom's exclusion row
// names are cleared from its mask row and the bits that are left counted.
__global__ void __launch_bounds__(32 * kListWarps)
k_list_count(int p0, int p1, ChunkMap map, const int *__restrict__ exclStart,
             const int *__restrict__ exclFlat, const int *__restrict__ flags, unsigned *masks,
             int *__restrict__ cnt, int *__restrict__ neighPair) {
  const int lane = threadIdx.x & 31;
  const int p = p0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (p >= min(p1, map.atoms()) || (*flags & FLAG_CELL)) return;
  const int i = map.atom(p);
  unsigned *row = masks + (size_t)(p - p0) * map.stride;
  const int cell = map.linkCells ? map.cellOf[i] : 0;
  const int nx = map.nlc[0], ny = map.nlc[1], nz = map.nlc[2];
  for (int e = exclStart[i] + lane; e < exclStart[i + 1]; e += 32) {
    const int j = exclFlat[e];
    if ((unsigned)j >= (unsigned)map.n) continue;
    if (!map.linkCells) {
      if (j > i) atomicAnd(row + (j >> 5), ~(1u << (j & 31)));
      continue;
    }
    const int kj = map.cellOf[j];
    if (kj < 0) continue;
    // offset of j's cell in the stencil, by the shorter way round
    int dx = kj % nx - cell % nx, dy = (kj / nx) % ny - (cell / nx) % ny,
        dz = kj / (nx * ny) - cell / (nx * ny);
    if (2 * dx > nx) dx -= nx; else if (2 * dx < -nx) dx += nx;
    if (2 * dy > ny) dy -= ny; else if (2 * dy < -ny) dy += ny;
    if (2 * dz > nz) dz -= nz; else if (2 * dz < -nz) dz += nz;
    if (abs(dx) > kMaxRatio || abs(dy) > kMaxRatio || abs(dz) > kMaxRatio) continue;
    const int l = c_stencilOf[((dz + kMaxRatio) * kInvSide + dy + kMaxRatio) * kInvSide + dx +
                              kMaxRatio];
    if (l < 0 || l >= map.cellCheck) continue;
    const int o = map.posOf[j] - map.cellStart[kj];
    atomicAnd(row + map.offsets(cell)[l] + (o >> 5), ~(1u << (o & 31)));
  }
  __syncwarp();
  int first, last, total = 0;
  map.range(p, cell, first, last);
  for (int c = first + lane; c < last; c += 32) total += __popc(__ldcg(row + c));
  total = __reduce_add_sync(0xffffffffu, total);
  if (lane == 0) {
    cnt[p] = total;
    neighPair[i] = total;
  }
}

// One warp per atom of [p0, p1): its entries at off[p], in bit order.  32
// words at a time are spread into shared memory, one lane per word, and
// copied out in consecutive addresses.
__global__ void __launch_bounds__(32 * kListWarps)
k_list_fill(int p0, int p1, ChunkMap map, const unsigned *__restrict__ masks,
            const long long *__restrict__ off, int *__restrict__ list) {
  __shared__ int buf[kListWarps][1024];
  const int lane = threadIdx.x & 31;
  const int p = p0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (p >= p1) return;
  int *const b = buf[threadIdx.x >> 5];
  const unsigned *row = masks + (size_t)(p - p0) * map.stride;
  const int cell = map.linkCells ? map.cellOf[map.order[p]] : 0;
  const int *bases =
      map.linkCells ? map.chunkBase + table_row(map.byStart, cell, map.cellStart) * map.stride
                    : nullptr;
  int first, last;
  map.range(p, cell, first, last);
  int *out = list + off[p];
  for (int c0 = first; c0 < last; c0 += 32) {
    const int c = c0 + lane;
    unsigned m = c < last ? row[c] : 0u;
    const int base = map.linkCells ? (c < last ? bases[c] : 0) : 32 * c;
    const int own = __popc(m);
    int x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int total = __shfl_sync(0xffffffffu, x, 31);
    for (int o = x; m;) {  // from the top bit down
      const int bit = 31 - __clz(m);
      m ^= 1u << bit;
      b[--o] = base + bit;
    }
    __syncwarp();
    for (int e = lane; e < total; e += 32) out[e] = map.linkCells ? map.order[b[e]] : b[e];
    __syncwarp();
    out += total;
  }
}

__global__ void k_gather_counts(int n, const int *__restrict__ order,
                                const int *__restrict__ neighPair, int *__restrict__ cnt) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) cnt[p] = neighPair[order[p]];
}

bool g_stencil_loaded[64];

int load_stencil() {
  int dev = 0;
  MDB_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && g_stencil_loaded[dev]) return MDBAS_NB_OK;
  int flat[LINK_STENCIL_MAX * 3];
  for (int l = 0; l < LINK_STENCIL_MAX; ++l)
    for (int d = 0; d < 3; ++d) flat[3 * l + d] = LINK_STENCIL[l][d];
  MDB_CUDA(cudaMemcpyToSymbol(c_stencil, flat, sizeof(flat)));
  short of[kInvSide * kInvSide * kInvSide];
  for (short &v : of) v = -1;
  for (int l = 0; l < LINK_STENCIL_MAX; ++l)
    of[((LINK_STENCIL[l][2] + kMaxRatio) * kInvSide + LINK_STENCIL[l][1] + kMaxRatio) * kInvSide +
       LINK_STENCIL[l][0] + kMaxRatio] = (short)l;
  MDB_CUDA(cudaMemcpyToSymbol(c_stencilOf, of, sizeof(of)));
  if (dev >= 0 && dev < 64) g_stencil_loaded[dev] = true;
  return MDBAS_NB_OK;
}

// Mask rows of at most this size are kept at a time; larger systems are
// tested in slabs of atoms, once to count and once to fill.
constexpr size_t kMaskBytes = (size_t)1 << 30;

// Bound of the FP32 test's error in r^2 near rl^2 when the coordinates' and
// shifts' roundings add up to `err` per axis (sum over the three axes by
// Cauchy-Schwarz, a quarter on top), with the roundings of the sum itself.
float test_band(double rl, double err) {
  return (float)(2.0 * 1.7320508 * rl * err * 1.25 + rl * rl / 2097152.0);
}

}  // namespace

int image_update_device(int n, const DevBox &b, double *x, double *y, double *z, cudaStream_t s) {
  if (n <= 0) return MDBAS_NB_OK;
  MDB_LAUNCH(k_image_update, grid_for(n, 256), 256, 0, s, n, b, x, y, z);
  return MDBAS_NB_OK;
}

int link_cell_dims(const DevBox &b, double cutOff, double delr, int linkRatio, int nlc[3]) {
  const double cutnb = cutOff + delr;
  nlc[0] = (int)(b.pa * (double)linkRatio / cutnb);
  nlc[1] = (int)(b.pb * (double)linkRatio / cutnb);
  nlc[2] = (int)(b.pc * (double)linkRatio / cutnb);
  return MDBAS_NB_OK;
}

int makelist_uses_link_cells(const DevBox &b, double cutOff, double delr, int linkRatio,
                             int noLink) {
  // makelist (src/list.c:40-57)
  int nlc[3];
  int r = linkRatio < 1 ? 1 : (linkRatio > 5 ? 5 : linkRatio);
  link_cell_dims(b, cutOff, delr, r, nlc);
  if (nlc[0] < 3 || nlc[1] < 3 || nlc[2] < 3) return 0;
  if (nlc[0] * nlc[1] * nlc[2] <= 27) return 0;
  if (noLink) return 0;
  return 1;
}

int build_ref_list(RefListWork &w, int n, const DevBox &b, double cutOff, double delr,
                   int linkRatio, int linkCells, const double *x, const double *y,
                   const double *z, const int *frozen, const int *exclStart,
                   const int *exclFlat, cudaStream_t s) {
  if (n <= 0) {
    w.entries = 0;
    return MDBAS_NB_OK;
  }
  const double cutnb = cutOff + delr;
  const double cutnb2 = cutnb * cutnb;
  const double ulp = 1.0 / 16777216.0;  // half an FP32 ulp, relative
  w.linkCells = linkCells;
  MDB_TRY(w.neighPair.ensure(sizeof(int) * n));
  MDB_TRY(w.order.ensure(sizeof(int) * n));
  MDB_TRY(w.cnt.ensure(sizeof(int) * n));
  // the flags (error bits, chunks needed) sit behind the entry total, so that
  // one copy brings back both
  MDB_TRY(w.off.ensure(sizeof(long long) * (n + 2)));
  int *flags = reinterpret_cast<int *>(w.off.as<long long>() + n + 1);
  MDB_TRY(w.cs.ensure(sizeof(float4) * n));

  ChunkMap map{};
  map.linkCells = linkCells;
  map.n = n;
  map.group = kGroup;
  int ratio = 1;
  if (linkCells) {
    MDB_TRY(load_stencil());
    ratio = linkRatio < 1 ? 1 : (linkRatio > kMaxRatio ? kMaxRatio : linkRatio);
    link_cell_dims(b, cutOff, delr, ratio, w.nlc);
    if (w.nlc[0] < 2 * ratio + 1 || w.nlc[1] < 2 * ratio + 1 || w.nlc[2] < 2 * ratio + 1)
      return MDBAS_NB_ERR_LINKCELL;  // LNKCELL_NCELLS_ERROR, src/list.c:1900-1908
    w.ncell = w.nlc[0] * w.nlc[1] * w.nlc[2];
    map.ncell = w.ncell;
    for (int d = 0; d < 3; ++d) map.nlc[d] = w.nlc[d];
    map.cellCheck = LINK_STENCIL_COUNT[ratio - 1];
    map.byStart = w.ncell > n;
    // chunks per cell of evenly spread atoms with room for fluctuations; a
    // denser cell reports what it needs and the build is made again
    const double per = (double)n / w.ncell;
    // Groups that mostly span cells are a warp's runs one after the other:
    // with few atoms and pieces they are split, until there are kTestWarps
    // warps (2,000 atoms spread over 100 A, link ratio 2: 204 -> 111 us, over
    // 200 A 144 -> 108; 3,000 atoms of water at ratio 5, where the pieces make
    // enough, would take 432 instead of 369)
    const double warps = n * std::max(1., map.cellCheck * std::min(1., per) / kPiece);
    while (map.group > 1 && warps < kTestWarps * map.group && per < map.group) map.group /= 2;
    map.stride = map.cellCheck * (int)((1.25 * per + 3. * sqrt(per)) / 32. + 1.);
    map.stride = (std::max(map.stride, w.maskStride) + 3) & ~3;
  } else {
    w.ncell = 0;
    map.stride = (((n + 31) >> 5) + 3) & ~3;
  }
  MDB_TRY(w.scanTmp.ensure(std::max(scan_tmp_bytes(w.ncell + 1), scan_tmp_bytes(n + 1))));
  const int ncell = w.ncell;
  const size_t tableRows = std::min(ncell, n);
  if (linkCells) {
    MDB_TRY(w.xu.ensure(sizeof(double) * n));
    MDB_TRY(w.yu.ensure(sizeof(double) * n));
    MDB_TRY(w.zu.ensure(sizeof(double) * n));
    MDB_TRY(w.xs.ensure(sizeof(double) * n));
    MDB_TRY(w.ys.ensure(sizeof(double) * n));
    MDB_TRY(w.zs.ensure(sizeof(double) * n));
    MDB_TRY(w.cellOf.ensure(sizeof(int) * n));
    MDB_TRY(w.posOf.ensure(sizeof(int) * n));
    MDB_TRY(w.tmpIdx.ensure(sizeof(int) * n));
    // counts and fill marks side by side: cleared together
    MDB_TRY(w.cellCount.ensure(sizeof(int) * 2 * (size_t)(ncell + 1)));
    MDB_TRY(w.cellStart.ensure(sizeof(int) * (ncell + 2)));
    MDB_TRY(w.chunkOff.ensure(sizeof(int) * tableRows * (map.cellCheck + 1)));
  }

  for (int attempt = 0;; ++attempt) {
    MDB_CUDA(cudaMemsetAsync(flags, 0, 2 * sizeof(int), s));
    float band, lx = 0.f, ly = 0.f, lz = 0.f;
    int exactOnly = 0;
    if (linkCells) {
      int *count = w.cellCount.as<int>(), *fill = count + ncell + 1;
      MDB_TRY(w.chunkBase.ensure(sizeof(int) * tableRows * map.stride));
      map.cellStart = w.cellStart.as<int>();
      map.cellOf = w.cellOf.as<int>();
      map.order = w.order.as<int>();
      map.posOf = w.posOf.as<int>();
      map.chunkOff = w.chunkOff.as<int>();
      map.chunkBase = w.chunkBase.as<int>();
      // coordinates up to two boxes (two roundings), the image shift and
      // its sum with a coordinate (up to three)
      const double ext = std::max({fabs(b.a1) + fabs(b.b1) + fabs(b.c1),
                                   fabs(b.a2) + fabs(b.b2) + fabs(b.c2),
                                   fabs(b.a3) + fabs(b.b3) + fabs(b.c3)});
      band = test_band(cutnb, (8. * ext + cutnb) * ulp);
      MDB_CUDA(cudaMemsetAsync(count, 0, sizeof(int) * 2 * (size_t)(ncell + 1), s));
      MDB_LAUNCH(k_lc_bin, grid_for(n, 256), 256, 0, s, n, b, w.nlc[0], w.nlc[1], w.nlc[2], x, y,
                 z, w.xu.as<double>(), w.yu.as<double>(), w.zu.as<double>(), w.cellOf.as<int>(),
                 count, flags);
      MDB_TRY(exclusive_scan32(count, w.cellStart.as<int>(), ncell, w.scanTmp.p, s));
      MDB_LAUNCH(k_lc_scatter, grid_for(n, 256), 256, 0, s, n, w.cellOf.as<int>(),
                 w.cellStart.as<int>(), fill, w.tmpIdx.as<int>());
      MDB_LAUNCH(k_lc_order, ncell, 256, 0, s, ncell, w.cellStart.as<int>(), w.tmpIdx.as<int>(),
                 w.order.as<int>());
      MDB_LAUNCH(k_lc_gather, grid_for(n, 256), 256, 0, s, ncell, b, w.cellStart.as<int>(),
                 w.order.as<int>(), w.xu.as<double>(), w.yu.as<double>(), w.zu.as<double>(),
                 frozen, w.xs.as<double>(), w.ys.as<double>(), w.zs.as<double>(),
                 w.cs.as<float4>(), w.posOf.as<int>());
      MDB_LAUNCH(k_lc_chunks, grid_for((long long)tableRows, kListWarps), 32 * kListWarps, 0, s,
                 ncell, w.nlc[0], w.nlc[1], w.nlc[2], map.cellCheck, map.stride, map.byStart,
                 w.cellStart.as<int>(), w.cellOf.as<int>(), w.order.as<int>(),
                 w.chunkOff.as<int>(), w.chunkBase.as<int>(), flags, flags + 1);
    } else {
      const double bx = b.a1, by = b.type == CUBIC ? b.a1 : b.b2,
                   bz = b.type == CUBIC ? b.a1 : b.c3;
      const double ux = b.u1, uy = b.type == CUBIC ? b.u1 : b.v2,
                   uz = b.type == CUBIC ? b.u1 : b.w3;
      // the FP32 minimum image is the orthorhombic box's
      exactOnly = !((b.type == CUBIC || b.type == ORBIC) && bx > 0. && by > 0. && bz > 0. &&
                    fabs(bx * ux - 1.) < 1e-9 && fabs(by * uy - 1.) < 1e-9 &&
                    fabs(bz * uz - 1.) < 1e-9);
      lx = (float)bx;
      ly = (float)by;
      lz = (float)bz;
      // two coordinates of half a box, their difference, the box length and
      // the difference from it
      band = test_band(cutnb, 4. * std::max({bx, by, bz}) * ulp);
      MDB_LAUNCH(k_vl_coords, grid_for(n, 256), 256, 0, s, n, bx, by, bz, x, y, z, frozen,
                 w.cs.as<float4>(), w.order.as<int>());
    }
    long long slab = (long long)(kMaskBytes / (sizeof(unsigned) * (size_t)map.stride)) &
                     ~(long long)(kGroup - 1);
    slab = std::max<long long>(slab, kGroup);
    const bool whole = slab >= n;
    MDB_TRY(w.masks.ensure(sizeof(unsigned) * (size_t)map.stride * std::min<long long>(slab, n)));
    const auto test = [&](int p0, int p1) -> int {
      unsigned *m = w.masks.as<unsigned>();
      const int g = grid_for(p1 - p0, map.group * kListWarps);
      if (linkCells) {
        const auto kern = frozen ? k_lc_masks<true> : k_lc_masks<false>;
        MDB_LAUNCH(kern, dim3(g, grid_for(map.stride, kPiece)), 32 * kListWarps, 0, s, p0, p1, b,
                   map, cutnb2, (float)cutnb2, band, w.xs.as<double>(), w.ys.as<double>(), w.zs.as<double>(), w.cs.as<float4>(),
                   flags, m);
      } else {
        const auto kern = frozen ? k_vl_masks<true> : k_vl_masks<false>;
        MDB_LAUNCH(kern, dim3(g, grid_for((n + 31) >> 5, kPiece)), 32 * kListWarps, 0, s, p0, p1,
                   b, map, cutnb2, (float)cutnb2, band, lx, ly, lz, exactOnly, x, y, z,
                   w.cs.as<float4>(), m);
      }
      MDB_LAUNCH(k_list_count, grid_for(p1 - p0, kListWarps), 32 * kListWarps, 0, s, p0, p1, map,
                 exclStart, exclFlat, flags, m, w.cnt.as<int>(), w.neighPair.as<int>());
      return MDBAS_NB_OK;
    };
    for (long long p = 0; p < n; p += slab) MDB_TRY(test((int)p, (int)std::min<long long>(p + slab, n)));
    MDB_TRY(exclusive_scan(w.cnt.as<int>(), w.off.as<long long>(), n, w.scanTmp.p, s));
    struct { long long total; int flags, need; } h;
    MDB_CUDA(cudaMemcpyAsync(&h, w.off.as<long long>() + n, sizeof(h), cudaMemcpyDeviceToHost, s));
    MDB_CUDA(cudaStreamSynchronize(s));
    if (h.flags & FLAG_NONFINITE) return MDBAS_NB_ERR_NONFINITE;
    if (h.flags & FLAG_OUTSIDE) return MDBAS_NB_ERR_BOX;
    if (h.flags & FLAG_CELL) {
      if (attempt > 0) return MDBAS_NB_ERR_CAPACITY;
      w.maskStride = map.stride = (h.need + 3) & ~3;
      continue;
    }
    w.entries = h.total;
    if (h.total > 0x7fffffffLL) return MDBAS_NB_ERR_CAPACITY;  // MDBas's int list index
    MDB_TRY(w.list.ensure(sizeof(int) * (size_t)std::max<long long>(h.total, 1)));
    for (long long p = 0; p < n; p += slab) {
      const int p0 = (int)p, p1 = (int)std::min<long long>(p + slab, n);
      if (!whole) MDB_TRY(test(p0, p1));
      MDB_LAUNCH(k_list_fill, grid_for(p1 - p0, kListWarps), 32 * kListWarps, 0, s, p0, p1, map,
                 w.masks.as<unsigned>(), w.off.as<long long>(), w.list.as<int>());
    }
    return MDBAS_NB_OK;
  }
}

int ref_list_offsets(RefListWork &w, int n, cudaStream_t s) {
  // Entry offsets of a list supplied by the caller (neighPair/order on the
  // device): exclusive scan of neighPair in neighOrder order.
  MDB_TRY(w.cnt.ensure(sizeof(int) * n));
  MDB_TRY(w.off.ensure(sizeof(long long) * (n + 1)));
  MDB_TRY(w.scanTmp.ensure(scan_tmp_bytes(n + 1)));
  MDB_LAUNCH(k_gather_counts, grid_for(n, 256), 256, 0, s, n, w.order.as<int>(),
             w.neighPair.as<int>(), w.cnt.as<int>());
  MDB_TRY(exclusive_scan(w.cnt.as<int>(), w.off.as<long long>(), n, w.scanTmp.p, s));
  return MDBAS_NB_OK;
}

}  // namespace mdbas
