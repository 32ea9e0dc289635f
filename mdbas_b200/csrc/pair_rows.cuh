// pair_rows.cuh -- the row walk of the FP64 pair kernels (pair_fp64.cu,
// adjoint.cu): one warp per atom i (in neighOrder position) over i's entries
// of the MDBas half list.
//
// Lanes read the entries of a row in consecutive addresses; the pairs inside
// the cut-off are queued in shared memory and handed to the caller 32 at a
// time, so the FP64 arithmetic runs with full warps (62% of a 14 A list lies
// within 12 A).  The walk is bound by latency: entries are loaded two rounds
// ahead and positions one round ahead (the 96,000-atom pair loop 0.93 -> 0.67
// ms, L2 warm), and atoms are handed out by a counter, the next one fetched while the
// current one runs.  A row can be cut into 2^split work items, so that a
// small system fills the SMs.
#pragma once

#include "common.cuh"

namespace mdbas {

constexpr int kRowWarps = 4;    // warps per block
constexpr int kRowQueue = 64;   // queued pairs per warp

// dist() of a pair whose displacement lies within half a box (times the
// margin) along every axis needs no image: nint() is 0 there and MDBas
// subtracts an exact zero.  The bounds are compared on the high words
// (0 for boxes without orthorhombic axes: always dist()).
struct NearBox {
  int hx, hy, hz;
};

__device__ __forceinline__ NearBox near_box(const DevBox &b) {
  if (b.type != CUBIC && b.type != ORBIC) return NearBox{0, 0, 0};
  return NearBox{__double2hiint(0.499 / fabs(b.u1)),
                 __double2hiint(0.499 / fabs(b.type == CUBIC ? b.u1 : b.v2)),
                 __double2hiint(0.499 / fabs(b.type == CUBIC ? b.u1 : b.w3))};
}

// dist(): minimum image in place, returns r^2.
__device__ __forceinline__ double near_dist(const DevBox &b, const NearBox &nb, double &dx,
                                            double &dy, double &dz) {
  if ((__double2hiint(dx) & 0x7fffffff) < nb.hx && (__double2hiint(dy) & 0x7fffffff) < nb.hy &&
      (__double2hiint(dz) & 0x7fffffff) < nb.hz)
    return dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
  return dist_d(b, dx, dy, dz);
}

struct HalfList {
  const int *order, *neighPair;
  const long long *off;
  const int *list;
};

// One warp's queue: displacement, r^2 and j.
struct RowQueue {
  double d[4][kRowQueue];
  int j[kRowQueue];
};

// begin(i) before a row; pairs(take, active, j, dx, dy, dz, r2) for up to 32
// pairs, called by the whole warp, active on the first `take` lanes; end(i)
// after it.  *work: zero before the launch.
template <class Begin, class Pairs, class End>
__device__ __forceinline__ void walk_rows(int n, int split, const DevBox &b, double cutOff2,
                                          const HalfList &hl, const double *__restrict__ x,
                                          const double *__restrict__ y,
                                          const double *__restrict__ z, RowQueue &queue,
                                          unsigned *work, Begin begin, Pairs pairs, End end) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const NearBox nb = near_box(b);
  unsigned next = 0;
  if (lane == 0) next = atomicAdd(work, 1u);
  for (;;) {
    const unsigned t = __shfl_sync(0xffffffffu, next, 0);
    if (t >= (unsigned)n << split) break;
    if (lane == 0) next = atomicAdd(work, 1u);
    const unsigned at = t >> split;
    const int i = hl.order[at];
    // this item's share of the row, in whole rounds of 32
    const long long all = hl.neighPair[i];
    const unsigned part = t & ((1u << split) - 1u);
    const int first = (int)((all * part) >> split) & ~31;
    const int cnt = (part + 1 == 1u << split ? (int)all : (int)((all * (part + 1)) >> split) & ~31) -
                    first;
    const int *row = hl.list + hl.off[at] + first;
    const double xi = x[i], yi = y[i], zi = z[i];
    begin(i);
    int jc = lane < cnt ? row[lane] : -1;
    int jn = 32 + lane < cnt ? row[32 + lane] : -1;
    double px = 0., py = 0., pz = 0.;
    const auto fetch = [&](int j) {
      if (j >= 0) {
        px = x[j];
        py = y[j];
        pz = z[j];
      }
    };
    fetch(jc);
    int qn = 0, k = 0;
    while (k < cnt || qn > 0) {
      while (k < cnt && qn < 32) {
        const int j = jc;
        double dx = px - xi, dy = py - yi, dz = pz - zi;
        k += 32;
        jc = jn;
        fetch(jc);
        jn = k + 32 + lane < cnt ? row[k + 32 + lane] : -1;
        const double r2 = near_dist(b, nb, dx, dy, dz);
        const bool in = j >= 0 && r2 <= cutOff2;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
          const int o = qn + __popc(m & lt);
          queue.d[0][o] = dx;
          queue.d[1][o] = dy;
          queue.d[2][o] = dz;
          queue.d[3][o] = r2;
          queue.j[o] = j;
        }
        qn += __popc(m);
      }
      __syncwarp();
      const int take = min(qn, 32);
      qn -= take;
      const int o = qn + lane;
      const bool active = lane < take;
      pairs(take, active, active ? queue.j[o] : 0, active ? queue.d[0][o] : 0.,
            active ? queue.d[1][o] : 0., active ? queue.d[2][o] : 0., active ? queue.d[3][o] : 1.);
      __syncwarp();  // the queue is read before the next round writes
    }
    end(i);
  }
}

// Blocks and row cuts of a walk over n atoms with `perSm` resident blocks.
// Fewer than two atoms per resident warp: rows cut in two (the pair loop of
// 3,000 atoms 52 -> 40 us, 6,000 65 -> 62; 12,000 100 -> 106, so not beyond).
struct RowGrid {
  int blocks, split;
};
inline RowGrid row_grid(int n, int perSm) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int most = sms * perSm;
  const int split = n < 2 * most * kRowWarps ? 1 : 0;
  const int need = grid_for((long long)n << split, kRowWarps);
  return RowGrid{need < most ? need : most, split};
}

}  // namespace mdbas
