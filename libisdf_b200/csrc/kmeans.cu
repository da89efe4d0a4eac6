// Density-weighted K-means interpolation-point selection on sm_100a.
//
// Reproduces the reference's CPU KMEAN (src/common/utility.cpp:631-988) bit
// for bit at one rank: every FP64 operation is an explicitly rounded add /
// sub / mul / div (no FMA contraction, like the reference's SSE2 x86-64
// build), the centroid sums are folded in point-index order per cluster, and
// every argmin keeps the first minimum. The reference's own GPU kernels
// (src/cuda/cuda_utils.cu:124-234,368-428) materialise an Npt x mu distance
// matrix and FMA-contract the distance; here the distance matrix is never
// stored and the arithmetic follows the CPU path.
//
// Device data layout (SoA, one entry per K-means point p in [0, Ng)):
//   pidx[p]   grid index of point p: the kept points ascending, then the
//             zero tail that aliases grid point 0 (utility.cpp:648,659,707);
//   px,py,pz  coordinates by the formula of utility.cpp:711-713;
//   pw        weight w[pidx[p]];
//   label[p]  nearest centroid.
// Centroids: double4 (x, y, z, 0) in cen[], rk on the device in st->rk.
#include <mutex>
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <optional>
#include <type_traits>
#include <vector>

#include "arena.h"
#include "comm.h"
#include "common.cuh"
#include "solve.h"
#include "kmeans.h"
#include "loop_graph.h"
#include "readback.h"

namespace isdf_b200 {

namespace {

constexpr int kTile = 2048;      // points per counting-sort tile (one walking warp each)
constexpr int kFinalChunk = 4096;  // points per partial argmin chunk
constexpr int kIterChunk = 8;    // Lloyd iterations launched between host checks (sharded)
constexpr int kBodyIters = 2;    // Lloyd iterations per graph of the loop
constexpr int kSlackIters = 1;   // ... behind the running one when the next graph is launched
constexpr int kAheadIters = 4;   // Lloyd iterations launched before the graph is made
constexpr int kMaxCellsPerDim = 20;  // centroid cell grid of the pruned assignment
constexpr int kMaxCells = kMaxCellsPerDim * kMaxCellsPerDim * kMaxCellsPerDim;

struct KmState {
  int s;        // Lloyd iterations begun (all of them completed when done)
  int flag;     // sharded: labels changed in the last assignment, over the ranks
  int changed;  // labels changed in the last assignment (n before the first iteration)
  int done;
  int rk;       // current number of centroids
  int npt;      // kept points
  int any_empty;
  int reset_bounds;  // centroid indices moved (empty-cluster compaction): bounds invalid
  unsigned long long maxw_bits;
  unsigned long long maxshift_bits;  // largest centroid move of this iteration (bit pattern)
  unsigned long long searches;       // assignments that ran the cell search (all iterations)
  unsigned ticket;  // blocks of k_hist_scan that have finished
  int rounds;       // iterations launched and begun, with those after the end
};

// ---------------------------------------------------------------- weight
// w(r) = 0 + (sum_{S2} psi^2) * (sum_{S1} psi^2), each sum a sequential fold
// over the states in increasing order (getpoints_Kmeans_MPI.cpp:37-45).
// One thread per grid point; a warp reads 32 consecutive doubles of a column.
__global__ void __launch_bounds__(256) k_weight(const double* __restrict__ psi, long long ng,
                                                int s2lo, int s2hi, int s1lo, int s1hi, int same,
                                                double* __restrict__ w) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < ng; r += stride) {
    const double* p = psi + r;
    double si = 0.0;
#pragma unroll 8
    for (int i = s2lo; i < s2hi; ++i) {
      double v = __ldg(p + (long long)i * ng);
      si = radd(si, rmul(v, v));
    }
    double sj = si;
    if (!same) {
      sj = 0.0;
#pragma unroll 8
      for (int j = s1lo; j < s1hi; ++j) {
        double v = __ldg(p + (long long)j * ng);
        sj = radd(sj, rmul(v, v));
      }
    }
    w[r] = radd(0.0, rmul(si, sj));
  }
}

// ---------------------------------------------------------------- filter
// maxW = max(0, max_r w(r)) (findMax starts at 0.0). Non-negative doubles
// order like their bit patterns, so an integer atomicMax is exact.
__global__ void k_maxw(const double* __restrict__ w, long long n, KmState* st) {
  double m = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    m = fmax(m, w[i]);
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.0)
    atomicMax(&st->maxw_bits, (unsigned long long)__double_as_longlong(m));
}

__device__ __forceinline__ bool kept(double wv, double thr) { return wv > thr; }

// Per-tile count of kept points (tile = blockDim.x * 4 points).
__global__ void __launch_bounds__(256) k_filter_count(const double* __restrict__ w, long long n,
                                                      const KmState* st, int* tile_cnt) {
  const double thr = rmul(1e-8, __longlong_as_double((long long)st->maxw_bits));
  __shared__ int warp_cnt[8];
  long long base = (long long)blockIdx.x * 1024;
  int c = 0;
  for (int k = 0; k < 4; ++k) {
    long long i = base + k * 256 + threadIdx.x;
    if (i < n && kept(w[i], thr)) ++c;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) warp_cnt[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int k = 0; k < 8; ++k) t += warp_cnt[k];
    tile_cnt[blockIdx.x] = t;
  }
}

// Exclusive scan of ntiles counts in one block; writes npt.
__global__ void __launch_bounds__(1024) k_scan_small(int* cnt, int ntiles, int* total) {
  __shared__ int part[1024];
  const int per = (ntiles + 1023) / 1024;
  const int lo = threadIdx.x * per, hi = min(lo + per, ntiles);
  int s = 0;
  for (int i = lo; i < hi; ++i) s += cnt[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    int v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int run = threadIdx.x ? part[threadIdx.x - 1] : 0;
  for (int i = lo; i < hi; ++i) {
    int v = cnt[i];
    cnt[i] = run;
    run += v;
  }
  if (threadIdx.x == 1023) *total = part[1023];
}

// Order-preserving compaction of the kept grid indices into pidx[0..npt);
// pidx[npt..n) was zeroed before (the reference's zero-initialised tail).
__global__ void __launch_bounds__(256) k_filter_scatter(const double* __restrict__ w, long long n,
                                                        const KmState* st, const int* tile_off,
                                                        int* __restrict__ pidx) {
  const double thr = rmul(1e-8, __longlong_as_double((long long)st->maxw_bits));
  __shared__ int warp_cnt[8][4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  long long base = (long long)blockIdx.x * 1024;
  unsigned ballots[4];
  for (int k = 0; k < 4; ++k) {
    long long i = base + k * 256 + threadIdx.x;
    bool f = i < n && kept(w[i], thr);
    ballots[k] = __ballot_sync(0xffffffffu, f);
    if (lane == 0) warp_cnt[wid][k] = __popc(ballots[k]);
  }
  __syncthreads();
  // order of elements: k-major, then warp, then lane
  int off = tile_off[blockIdx.x];
  for (int k = 0; k < 4; ++k) {
    int before = 0;
    for (int kk = 0; kk < k; ++kk)
      for (int ww = 0; ww < 8; ++ww) before += warp_cnt[ww][kk];
    for (int ww = 0; ww < wid; ++ww) before += warp_cnt[ww][k];
    long long i = base + k * 256 + threadIdx.x;
    if (ballots[k] & (1u << lane)) {
      int r = __popc(ballots[k] & ((1u << lane) - 1u));
      pidx[off + before + r] = (int)i;
    }
  }
}

// Coordinates of grid point t by the formula of utility.cpp:711-713 (and
// :758-760 for centroids), each operation rounded as the reference's build.
__device__ __forceinline__ void grid_coords(int t, int nx, int ny, double dx0, double dx1,
                                            double dx2, double* gx_, double* gy_,
                                            double* gz_) {
  const double gx = rmul((double)(t % nx), dx0);
  const double gy = rmul(rdiv(rsub((double)(t % (nx * ny)), rdiv(gx, dx0)), (double)nx), dx1);
  const double gz =
      rmul(rdiv(rsub(rsub((double)t, rdiv(gx, dx0)), rmul(rdiv(gy, dx1), (double)nx)),
                (double)(nx * ny)),
           dx2);
  *gx_ = gx;
  *gy_ = gy;
  *gz_ = gz;
}

// Point coordinates and weights (utility.cpp:707-713); the centroids start
// at the first rk kept points (utility.cpp:750-762), i.e. points 0..rk-1.
__global__ void k_points(const int* __restrict__ pidx, const double* __restrict__ w, int n,
                         int nx, int ny, double dx0, double dx1, double dx2,
                         double* __restrict__ px, double* __restrict__ py,
                         double* __restrict__ pz, double* __restrict__ pw, int rk,
                         double4* __restrict__ cen) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    int t = pidx[p];
    double gx, gy, gz;
    grid_coords(t, nx, ny, dx0, dx1, dx2, &gx, &gy, &gz);
    px[p] = gx;
    py[p] = gy;
    pz[p] = gz;
    pw[p] = w[t];
    if (p < rk) cen[p] = make_double4(gx, gy, gz, 0.0);
  }
}

// Warm start (utility.cpp:725-749): w at the previous pivots, for the
// filter test the reference applies to them.
__global__ void k_gather_w(const double* __restrict__ w, const int* __restrict__ idx, int cnt,
                           double* __restrict__ out) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt; j += gridDim.x * blockDim.x)
    out[j] = w[idx[j]];
}

// Warm start: centroid j starts at grid point cinit[j].
__global__ void k_warm_centroids(const int* __restrict__ cinit, int rk, int nx, int ny,
                                 double dx0, double dx1, double dx2,
                                 double4* __restrict__ cen) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < rk; j += gridDim.x * blockDim.x) {
    double gx, gy, gz;
    grid_coords(cinit[j], nx, ny, dx0, dx1, dx2, &gx, &gy, &gz);
    cen[j] = make_double4(gx, gy, gz, 0.0);
  }
}

// ---------------------------------------------------------------- assign
// d = ((dx*dx + dy*dy) + dz*dz) with dx = point - centroid (pdist2,
// utility.cpp:598-615); label = first centroid reaching the minimum
// (findMin Dim=1, utility.cpp:579-595).
constexpr int kAssignThreads = 128;

// ---------------------------------------------------------------- pruned assign
// Exact spatial pruning: centroids are binned into a uniform nc^3 cell grid
// over the box, and a search leaves out a cell only when the squared distance
// from the points to the cell's box (widened by tol), shrunk by a relative
// 2e-14 safety factor (well above the rounding of both the box bound and the
// distance formula), is strictly greater than a distance already found. Every
// centroid left out would have computed a strictly larger distance, so the
// result - the first centroid in index order reaching the minimum computed
// distance, compared as (d, index) pairs - is the brute-force result bit for
// bit.
struct CellGrid {
  int nc;
  double h[3];
  double inv_h[3];  // (a cell found with it is off by rounding only, far inside tol)
  double tol;
};

// Thread -> point map of the assignment. Brick mode: each warp takes a
// 4 x 4 x 2 brick of grid points instead of 32 points along the kept-point
// list, so that its lanes search nearly the same cells; a grid point that
// the weight filter dropped leaves its lane idle (g2p[g] = -1), and the
// zero-tail points p >= npt (copies of grid point 0) follow the bricks one
// per thread. Linear mode: thread t takes point t. Either way every point is
// assigned once and the result does not depend on the map.
// A rank of a sharded selection assigns only its points [p_lo, p_hi): its
// kept points lie in a z range of bricks (launched from brick thread t0 on),
// its zero-tail points follow them.
struct AssignMap {
  int brick;  // 0: linear
  int nx, ny, nz;
  int nbx, nby;    // bricks along x and y
  long long nbt;   // brick threads launched: bricks x 32
  long long t0;    // first brick thread
  int npt, n;
  int p_lo, p_hi;  // the points this launch assigns
  const int* g2p;  // grid index -> kept-point index (or -1); nullptr: identity
};

// One selection as the kernels of a Lloyd iteration see it: every buffer is the
// selection's own. The kernels take a batch of them by value and a job per
// blockIdx.y, its grid sized for the largest: one selection alone (N = 1), or
// the small ones of a batch side by side, which leave most of the GPU idle one
// by one.
struct KmJob {
  const int* pidx;
  const double *px, *py, *pz;
  int* label;
  int n;
  double4 *sorted, *cen, *sums;
  int *hist, *members, *start;
  double2* bnd;
  double* shift;
  float* nbshift;
  KmState* st;
  int* cell_start;
  double4* cell_cen;
  int* cell_of;
  const int* pcell;
  const double2* pd12;
  CellGrid cg;
  AssignMap am;
  // the points folded into the sums: all of them, or a rank's own in a sharded
  // selection, whose partial sums go elsewhere and decide nothing by themselves
  const int* f_label;
  const double *fx, *fy, *fz, *fw;
  int f_n, f_npt;  // how many, and how many of them are kept points
  double4* f_sums;
  int sharded;
  int* sel;      // grid index of the nearest point to each centroid
  double dx[3];  // grid spacings
  double max_f;  // the loop goes on while more labels than this change
  int max_iter;
};

constexpr int kBatchJobs = kKmeansBatchGroup;  // selections per launch (6.5 KB of parameters)
template <int N>
struct KmJobs {
  KmJob j[N];
};

__device__ __forceinline__ int assign_point(long long t, const AssignMap& am) {
  if (!am.brick) {
    const long long p = am.p_lo + t;
    return p < am.p_hi ? (int)p : -1;
  }
  if (t >= am.nbt) {
    const long long p = (long long)max(am.npt, am.p_lo) + (t - am.nbt);
    return p < am.p_hi ? (int)p : -1;
  }
  t += am.t0;
  const long long b = t >> 5;
  const int l = (int)(t & 31);
  const int bx = (int)(b % am.nbx);
  const long long r = b / am.nbx;
  const int by = (int)(r % am.nby), bz = (int)(r / am.nby);
  const int ix = bx * 4 + (l & 3), iy = by * 4 + ((l >> 2) & 3), iz = bz * 2 + (l >> 4);
  if (ix >= am.nx || iy >= am.ny || iz >= am.nz) return -1;
  const int g = ix + am.nx * (iy + am.ny * iz);
  const int p = am.g2p ? am.g2p[g] : g;
  return (p >= am.p_lo && p < am.p_hi) ? p : -1;
}

// Inverse of the kept-point list: g2p[pidx[p]] = p for p < npt (the rest -1).
__global__ void k_grid_to_point(const int* __restrict__ pidx, int npt, int* __restrict__ g2p) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npt; p += gridDim.x * blockDim.x)
    g2p[pidx[p]] = p;
}

// In-place inclusive scan of a[0..n) by a block of 1024 threads: every
// thread sums a contiguous chunk, the chunk totals are scanned across the
// warp and the block, and each thread rewrites its chunk.
__device__ void block_inclusive_scan(int* a, int n, int* warp_tot) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int per = (n + 1023) / 1024;
  const int b0 = min(n, tid * per), b1 = min(n, b0 + per);
  int sum = 0;
  for (int i = b0; i < b1; ++i) sum += a[i];
  int v = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) warp_tot[w] = v;
  __syncthreads();
  if (w == 0) {
    int t = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += u;
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  int run = v - sum + (w > 0 ? warp_tot[w - 1] : 0);
  for (int i = b0; i < b1; ++i) {
    run += a[i];
    a[i] = run;
  }
  __syncthreads();
}

// Squared distance in the reference's rounding (pdist2, utility.cpp:598-615).
__device__ __forceinline__ double ref_dist2(double x, double y, double z, const double4& c) {
  const double d1 = rsub(x, c.x), d2 = rsub(y, c.y), d3 = rsub(z, c.z);
  return radd(radd(rmul(d1, d1), rmul(d2, d2)), rmul(d3, d3));
}

// Distance bounds (Hamerly): bnd[p] = (u, l), u >= the true distance from p
// to its assigned centroid, l <= the true distance to every other centroid.
// Moving centroids move them by at most shift[label] and the largest shift.
// When u (1 + 1e-12) < l, the assigned centroid is strictly nearest with a
// margin far above the relative error of the rounded squared distances
// (~1e-15), so the reference's argmin (first minimum of the rounded
// distances) is the assigned label and the search is skipped. Otherwise the
// search runs and the bounds are rebuilt from it: u from the best distance, l
// from the second best seen and the radius searched.
constexpr double kBoundMargin = 1.0 + 1e-12;
constexpr double kRoundUp = 1.0 + 1e-13;
constexpr double kRoundDown = 1.0 - 1e-13;

// Per point, once per selection (the points do not move): its cell and the
// distances from it to the outside of the 3^3 and 5^3 cell blocks around it
// (rounded down, less the binning tolerance; infinite where a block reaches
// the domain's faces), which the distance-bound test reads instead of
// recomputing three divisions and twelve face distances every iteration.
__global__ void k_point_cells(const double* __restrict__ px, const double* __restrict__ py,
                              const double* __restrict__ pz, int n, CellGrid g,
                              int* __restrict__ pcell, double2* __restrict__ pd12) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double x = px[p], y = py[p], z = pz[p];
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  const int pi = min(g.nc - 1, max(0, (int)floor(x / g.h[0])));
  const int pj = min(g.nc - 1, max(0, (int)floor(y / g.h[1])));
  const int pk = min(g.nc - 1, max(0, (int)floor(z / g.h[2])));
  double D1 = inf, D2 = inf;
  if (pi >= 2) D1 = fmin(D1, x - (pi - 1) * g.h[0]);
  if (pi + 2 <= g.nc - 1) D1 = fmin(D1, (pi + 2) * g.h[0] - x);
  if (pj >= 2) D1 = fmin(D1, y - (pj - 1) * g.h[1]);
  if (pj + 2 <= g.nc - 1) D1 = fmin(D1, (pj + 2) * g.h[1] - y);
  if (pk >= 2) D1 = fmin(D1, z - (pk - 1) * g.h[2]);
  if (pk + 2 <= g.nc - 1) D1 = fmin(D1, (pk + 2) * g.h[2] - z);
  if (pi >= 3) D2 = fmin(D2, x - (pi - 2) * g.h[0]);
  if (pi + 3 <= g.nc - 1) D2 = fmin(D2, (pi + 3) * g.h[0] - x);
  if (pj >= 3) D2 = fmin(D2, y - (pj - 2) * g.h[1]);
  if (pj + 3 <= g.nc - 1) D2 = fmin(D2, (pj + 3) * g.h[1] - y);
  if (pk >= 3) D2 = fmin(D2, z - (pk - 2) * g.h[2]);
  if (pk + 3 <= g.nc - 1) D2 = fmin(D2, (pk + 3) * g.h[2] - z);
  pcell[p] = pi + g.nc * (pj + g.nc * pk);
  pd12[p] = make_double2(D1 * kRoundDown - g.tol, D2 * kRoundDown - g.tol);
}

// Warp-coherent search. A warp's points are a 4 x 4 x 2 brick of the grid
// (or 32 consecutive points), so the points of a warp that fail the bound
// test share their candidates: with U the largest of their seed distances
// (squared distance to the old label, which bounds each one's nearest), every
// centroid that can be nearest to one of them lies within sqrt(U) of the
// points' bounding box. The cells of one (y, z) row are contiguous in cell
// order, so the lanes take a row each, then the rows' centroids 32 at a time:
// those within sqrt(U) of the box go to shared memory as single-precision
// offsets c from the box's centre, (-2 c, |c|^2), kWarpCand at most before they
// are scanned (any number of cells and candidates is taken in such portions).
// The scan keeps the two smallest |c|^2 - 2 p.c per point, the squared distance
// less |p|^2 in three multiply-adds. Their error against the exact distance is
// below err = 2^-18 r^2, r = sqrt(U) + h and h the box's half diagonal (all
// offsets are at most r long; rounding both, |c|^2, |p|^2 and the three sums
// comes to 22 2^-24 r^2 with the worst signs), so when the second is more than
// 2 err above the first, the first is the only candidate
// that can be the portion's nearest, and its distance alone is computed in the
// reference's rounding; otherwise every candidate within 2 err of the smallest
// is. Distances so computed are compared as (d, index) pairs: the label is
// brute force's bit for bit. All other candidates are farther than the second
// smallest less err, and centroids not staged farther than sqrt(U): the lower
// bound.
// What this replaced: FP64 distances to every candidate, and a per-point search
// in rings of cells where a warp had more than 216 cells or 160 candidates (a
// few warps in the sparse regions, which the launch then waited for) or, in the
// first assignment, no seed. A launch late in a selection: 64 000 points and
// 309 centroids 47 -> 10 us, 151 875 and 505 68 -> 18 us, 884 736 and 2979
// 140 -> 55 us; the first assignment of the last 9200 -> 510 us.
constexpr int kWarpCand = 128;   // candidates staged per warp

// The warp's least float / largest float / largest non-negative float, by the
// integer reductions (a float's bits, the negative ones' magnitude flipped, order as
// the values do).
__device__ __forceinline__ int float_order(float v) {
  const int i = __float_as_int(v);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float order_float(int i) {
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}
__device__ __forceinline__ double warp_least(bool in, double v) {
  const int i = in ? float_order(__double2float_rd(v)) : 0x7fffffff;
  return (double)order_float(__reduce_min_sync(0xffffffffu, i));
}
__device__ __forceinline__ double warp_most(bool in, double v) {
  const int i = in ? float_order(__double2float_ru(v)) : (int)0x80000000;
  return (double)order_float(__reduce_max_sync(0xffffffffu, i));
}

// A seed for the first assignment. The centroids start at the first rk points
// of the list, which fill the lowest planes and rows of the box: the nearest
// is above, below or beside the point itself. (Any centroid is a valid seed.)
__device__ __forceinline__ int first_seed(int p, int rk, const int* __restrict__ pidx,
                                          const AssignMap& am) {
  if (p < rk) return p;
  if (!am.brick) return rk - 1;
  const int t = pidx[p], last = pidx[rk - 1], plane = am.nx * am.ny;
  int g = t % plane;                  // the point's column in the lowest plane
  const int top = last / plane;       // the plane the centroids end in
  if (top > 0) {
    g += (g + top * plane <= last ? top : top - 1) * plane;
  } else if (g > last) {              // beyond the rows they cover
    const int row = last / am.nx;
    g = g % am.nx + am.nx * (row > 0 ? row - 1 : 0);
    if (g > last) g = last;
  }
  const int j = am.g2p ? am.g2p[g] : g;
  return j >= 0 && j < rk ? j : rk - 1;
}

template <int N>
__global__ void __launch_bounds__(kAssignThreads, 8)
    k_assign_warp(const __grid_constant__ KmJobs<N> JS, int count) {
  after_previous();
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  KmState* st = J.st;
  if (st->done) return;
  const double *px = J.px, *py = J.py, *pz = J.pz;
  const double4 *cen = J.cen, *cell_cen = J.cell_cen;
  const int* cell_start = J.cell_start;
  const CellGrid& g = J.cg;
  int* label = J.label;
  double2* bnd = J.bnd;
  __shared__ float4 cand[kAssignThreads / 32][kWarpCand];  // -2 c, |c|^2
  __shared__ int cand_at[kAssignThreads / 32][kWarpCand];  // place in cell_cen
  const int rk = st->rk;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int p = assign_point((long long)blockIdx.x * blockDim.x + threadIdx.x, J.am);
  bool need = false;
  int old = -1;
  if (p >= 0 && p < J.n) {
    old = count ? label[p] : -1;
    need = true;
    if (old >= 0 && old < rk && count && !st->reset_bounds) {
      const double2 b = bnd[p];
      // Every other centroid moved closer by at most its shift: at most
      // the 3^3-block maximum inside the 27 cells around p, the 5^3-block
      // maximum in the ring beyond (which started at least D1 = dd.x away),
      // the global maximum further out (at least D2 = dd.y away); no bound
      // across the domain's faces.
      const double gmax = __longlong_as_double((long long)st->maxshift_bits);
      const int cell = J.pcell[p];
      const double near1 = (double)J.nbshift[cell], near2 = (double)J.nbshift[kMaxCells + cell];
      const double2 dd = J.pd12[p];
      double lo = __dsub_rd(b.y, near1);
      lo = fmin(lo, __dsub_rd(fmax(b.y, dd.x), near2));
      lo = fmin(lo, __dsub_rd(fmax(b.y, dd.y), gmax));
      lo = fmax(0.0, lo);
      double up = __dadd_ru(b.x, J.shift[old]);
      if (!(up * kBoundMargin < lo))
        up = __dmul_ru(__dsqrt_ru(ref_dist2(px[p], py[p], pz[p], cen[old])), kRoundUp);
      if (up * kBoundMargin < lo) {  // the label stays
        bnd[p] = make_double2(up, lo);
        need = false;
      }
    }
  }
  const unsigned mask = __ballot_sync(0xffffffffu, need);
  if (!mask) return;
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  double x = 0.0, y = 0.0, z = 0.0, best = 0.0;
  int bj = 0;
  if (need) {
    x = px[p];
    y = py[p];
    z = pz[p];
    bj = old >= 0 && old < rk ? old : first_seed(p, rk, J.pidx, J.am);
    best = ref_dist2(x, y, z, cen[bj]);
  }
  const double shrink = 1.0 - 2e-14;
  // (all rounded outward to single precision: what they bound stays bounded)
  const double U = warp_most(true, best);  // 0 on the lanes that do not search
  const double x0 = warp_least(need, x), x1 = warp_most(need, x);
  const double y0 = warp_least(need, y), y1 = warp_most(need, y);
  const double z0 = warp_least(need, z), z1 = warp_most(need, z);
  const double xc = 0.5 * (x0 + x1), yc = 0.5 * (y0 + y1), zc = 0.5 * (z0 + z1);
  const double R = __dmul_ru(__dsqrt_ru(U), kRoundUp) + g.tol;
  const float fx = (float)(x - xc), fy = (float)(y - yc), fz = (float)(z - zc);
  const float pp = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
  const float hx = __double2float_ru(x1 - xc), hy = __double2float_ru(y1 - yc),
              hz = __double2float_ru(z1 - zc);
  const double reach = R + (x1 - xc) + (y1 - yc) + (z1 - zc);  // >= sqrt(U) + h
  // (the last term covers products below the normal range)
  const float err = __double2float_ru(3.814697265625e-6 * reach * reach) + 1e-37f;
  const float far = __double2float_ru(U) + 2.0f * err;  // beyond: more than sqrt(U) from the box
  const int nc = g.nc;
  const int i0 = min(nc - 1, max(0, (int)floor((x0 - R) * g.inv_h[0])));
  const int i1 = min(nc - 1, max(0, (int)floor((x1 + R) * g.inv_h[0])));
  const int j0 = min(nc - 1, max(0, (int)floor((y0 - R) * g.inv_h[1])));
  const int j1 = min(nc - 1, max(0, (int)floor((y1 + R) * g.inv_h[1])));
  const int k0 = min(nc - 1, max(0, (int)floor((z0 - R) * g.inv_h[2])));
  const int k1 = min(nc - 1, max(0, (int)floor((z1 + R) * g.inv_h[2])));
  const int nj = j1 - j0 + 1, nrow = nj * (k1 - k0 + 1);
  float4* cw = cand[wid];
  int* cat = cand_at[wid];
  double second = inf;
  // the nearest of the candidates staged, into (best, bj) and second
  auto scan = [&](int total) {
    if (!need) return;
    const float finf = __int_as_float(0x7f800000);
    float m1 = finf, m2 = finf;
    int q1 = 0;
#pragma unroll 4
    for (int q = 0; q < total; ++q) {
      const float4 c = cw[q];
      const float d = fmaf(fx, c.x, fmaf(fy, c.y, fmaf(fz, c.z, c.w)));
      m2 = fminf(m2, fmaxf(m1, d));
      q1 = d < m1 ? q : q1;
      m1 = fminf(m1, d);
    }
    auto consider = [&](int q) {
      const double4 c = cell_cen[cat[q]];
      const double d = ref_dist2(x, y, z, c);
      const int j = (int)c.w;
      if (d < best || (d == best && j < bj)) {
        if (j != bj) second = fmin(second, best);
        best = d;
        bj = j;
      } else if (j != bj) {
        second = fmin(second, d);
      }
    };
    const float thr = m1 + 2.0f * err;
    if (m2 > thr) {
      consider(q1);
      second = fmin(second, fmax(0.0, (double)m2 + (double)pp - (double)err));
    } else {
      float next = finf;  // the smallest distance left out
      for (int q = 0; q < total; ++q) {
        const float4 c = cw[q];
        const float d = fmaf(fx, c.x, fmaf(fy, c.y, fmaf(fz, c.z, c.w)));
        if (!(d > thr)) consider(q);
        else next = fminf(next, d);
      }
      second = fmin(second, fmax(0.0, (double)next + (double)pp - (double)err));
    }
  };
  int total = 0;
  for (int base = 0; base < nrow; base += 32) {
    // one (y, z) row of cells per lane: its centroids are contiguous
    int cnt = 0, first = 0;
    if (base + lane < nrow) {
      const int cj = j0 + (base + lane) % nj, ck = k0 + (base + lane) / nj;
      // distance from the points' box to the row's (widened by tol)
      const double by = fmax(0.0, fmax(cj * g.h[1] - g.tol - y1, y0 - (cj + 1) * g.h[1] - g.tol));
      const double bz = fmax(0.0, fmax(ck * g.h[2] - g.tol - z1, z0 - (ck + 1) * g.h[2] - g.tol));
      if (!((by * by + bz * bz) * shrink > U)) {
        const int id = nc * (cj + nc * ck);
        first = cell_start[id + i0];
        cnt = cell_start[id + i1 + 1] - first;
      }
    }
    int off = cnt;  // inclusive scan over the warp
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += v;
    }
    const int here = __shfl_sync(0xffffffffu, off, 31);
    for (int e0 = 0; e0 < here; e0 += 32) {
      const int e = e0 + lane;
      // the row of ordinal e: the first lane whose inclusive count exceeds it
      int lo = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int v = __shfl_sync(0xffffffffu, off, lo + step - 1);
        if (v <= e) lo += step;
      }
      const int at = __shfl_sync(0xffffffffu, first, lo & 31) + e -
                     (__shfl_sync(0xffffffffu, off, lo & 31) - __shfl_sync(0xffffffffu, cnt, lo & 31));
      bool in = false;
      float cx = 0.f, cy = 0.f, cz = 0.f;
      if (e < here) {
        const double4 c = cell_cen[at];
        cx = (float)(c.x - xc);
        cy = (float)(c.y - yc);
        cz = (float)(c.z - zc);
        const float bx = fmaxf(0.f, fabsf(cx) - hx), by = fmaxf(0.f, fabsf(cy) - hy),
                    bz = fmaxf(0.f, fabsf(cz) - hz);
        in = !(fmaf(bx, bx, fmaf(by, by, bz * bz)) > far);
      }
      const unsigned got = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int to = total + __popc(got & ((1u << lane) - 1u));
        cw[to] = make_float4(-2.f * cx, -2.f * cy, -2.f * cz, fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
        cat[to] = at;
      }
      total += __popc(got);
      if (total > kWarpCand - 32) {
        __syncwarp();
        scan(total);
        __syncwarp();
        total = 0;
      }
    }
  }
  __syncwarp();
  if (total > 0) scan(total);
  int changed = 0;
  if (need) {
    // every centroid not staged is more than sqrt(U) from the point
    const double floor2 = U * shrink;
    bnd[p] = make_double2(__dmul_ru(__dsqrt_ru(best), kRoundUp),
                          __dmul_rd(__dsqrt_rd(fmin(second, floor2)), kRoundDown));
    if (count && old != bj) ++changed;
    label[p] = bj;
  }
  for (int o = 16; o > 0; o >>= 1) changed += __shfl_xor_sync(0xffffffffu, changed, o);
  if (lane == 0) {
    if (count && changed) atomicAdd(&st->changed, changed);
    atomicAdd(&st->searches, (unsigned long long)__popc(mask));
  }
}

// ---------------------------------------------------------------- control
// The loop test of utility.cpp:812. Every kernel up to the last block of
// k_hist_scan, which begins the iteration, finds it by itself.
__device__ __forceinline__ bool goes_on(const KmJob& J) {
  return J.sharded || ((double)J.st->changed > J.max_f && J.st->s < J.max_iter);
}

// ---------------------------------------------------------------- update
// Stable counting sort of the points by label (tiles of kTile points), then
// one warp per cluster and component folds w, w*x, w*y, w*z over the members
// in increasing point index: the exact sequence of additions of
// utility.cpp:816-822.
template <int N>
__global__ void __launch_bounds__(256) k_hist(const __grid_constant__ KmJobs<N> JS, const LoopSignal sig) {
  after_previous();
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  KmState* st = J.st;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const int rounds = ++st->rounds;
    if (blockIdx.y == 0) loop_round(sig, rounds);
  }
  if (st->done || !goes_on(J) || blockIdx.x * kTile >= J.f_n) return;
  extern __shared__ int sh[];
  const int rk = st->rk;
  for (int l = threadIdx.x; l < rk; l += blockDim.x) sh[l] = 0;
  __syncthreads();
  const int base = blockIdx.x * kTile;
  const int end = min(base + kTile, J.f_n);
  for (int p = base + threadIdx.x; p < end; p += blockDim.x) atomicAdd(&sh[J.f_label[p]], 1);
  __syncthreads();
  int* row = J.hist + (size_t)blockIdx.x * rk;
  for (int l = threadIdx.x; l < rk; l += blockDim.x) row[l] = sh[l];
}

// Per label: exclusive scan over tiles (in place) and the member count. A
// block holds 32 labels (one per lane) and kScanWarps warps, each over a
// contiguous range of tiles: the warps' range sums, their exclusive prefix in
// shared memory, then each warp rewrites its range from that prefix. One
// thread per label walking all tiles left the scan bound by the latency of
// its ~ntiles/16 dependent load batches. The last block to finish scans the
// member counts into each label's first slot and begins the iteration: one
// launch where three single-block kernels ran. The last selection of a batch to
// stop (live: how many still run; nullptr for one alone) ends the loop.
constexpr int kScanWarps = 16;

template <int N>
__global__ void __launch_bounds__(32 * kScanWarps)
    k_hist_scan(const __grid_constant__ KmJobs<N> JS, const LoopSignal sig, int* live) {
  after_previous();
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  KmState* st = J.st;
  if (st->done) return;
  if (!goes_on(J)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->done = 1;
      if (!live || atomicSub(live, 1) == 1) loop_over(sig);
    }
    return;
  }
  const int rk = st->rk;
  const int ntiles = (J.f_n + kTile - 1) / kTile;
  int* hist = J.hist;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int l = blockIdx.x * 32 + lane;
  const int per = (ntiles + kScanWarps - 1) / kScanWarps;
  const int t0 = w * per, t1 = min(t0 + per, ntiles);
  __shared__ int part[kScanWarps][32];
  __shared__ bool last;
  // kB tiles of a warp's range are held at once, their loads all ahead of the sums
  auto scan = [&](auto held) {
    constexpr int kB = decltype(held)::value;
    int v[kB];
    auto load = [&](int t) {
#pragma unroll
      for (int u = 0; u < kB; ++u) v[u] = t + u < t1 ? hist[(size_t)(t + u) * rk + l] : 0;
    };
    int sum = 0;
    if (l < rk) {
      for (int t = t0; t < t1; t += kB) {
        load(t);
#pragma unroll
        for (int u = 0; u < kB; ++u) sum += v[u];
      }
    }
    part[w][lane] = sum;
    __syncthreads();
    if (l < rk) {
      int run = 0;
      for (int q = 0; q < w; ++q) run += part[q][lane];
      for (int t = t0; t < t1; t += kB) {
        if (per > kB) load(t);  // else still there
#pragma unroll
        for (int u = 0; u < kB; ++u) {
          if (t + u < t1) hist[(size_t)(t + u) * rk + l] = run;
          run += v[u];
        }
      }
      // the last warp's prefix covers every tile (its own range may be empty)
      if (w == kScanWarps - 1) J.members[l] = run;
    }
  };
  if (per <= 4) scan(std::integral_constant<int, 4>());
  else scan(std::integral_constant<int, 16>());
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  // exclusive scan of the member counts: start[l] (staged in shared memory: a
  // thread walking its labels in global memory waits for each)
  __threadfence();
  extern __shared__ int mem[];  // rk counts
  for (int i = threadIdx.x; i < rk; i += 32 * kScanWarps) mem[i] = __ldcg(J.members + i);
  __syncthreads();
  const int each = (rk + 32 * kScanWarps - 1) / (32 * kScanWarps);
  const int lo = min(rk, (int)threadIdx.x * each), hi = min(rk, lo + each);
  int mine = 0;
  for (int i = lo; i < hi; ++i) mine += mem[i];
  int inc = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  int* tot = part[0];
  if (lane == 31) tot[w] = inc;
  __syncthreads();
  int run = inc - mine;
  for (int q = 0; q < w; ++q) run += tot[q];
  for (int i = lo; i < hi; ++i) {
    const int v = mem[i];
    mem[i] = run;
    run += v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rk; i += 32 * kScanWarps) J.start[i] = mem[i];
  if (threadIdx.x == 0) {
    st->ticket = 0;
    if (!J.sharded) {
      st->s += 1;
      st->changed = 0;
      st->any_empty = 0;
      st->reset_bounds = 0;
      st->maxshift_bits = 0;
    }
  }
}

// The points' (w x, w y, w z, w) into cluster order, so that the per-cluster
// fold reads its members contiguously. One tile per block, a stretch of
// kTile / 8 consecutive points per warp: each warp counts its points per label
// (peers with equal labels in 32 points make one addition), the counts become
// each warp's offset within the tile, and each warp then gives its points their
// stable places and moves them. The walks of eight warps run side by side: one
// warp walking the whole tile took 15 us of a 98 us iteration at 64 000 points
// whatever their number, and this takes 5.
constexpr int kScatterWarps = 8;

template <int N>
__global__ void __launch_bounds__(32 * kScatterWarps)
    k_scatter(const __grid_constant__ KmJobs<N> JS) {
  after_previous();
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  const KmState* st = J.st;
  if (st->done || blockIdx.x * kTile >= J.f_n) return;
  extern __shared__ __align__(16) unsigned short cnt[];  // [label][warp]
  const int rk = st->rk;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int kPer = kTile / kScatterWarps, kSteps = kPer / 32;
  uint4* cnt4 = reinterpret_cast<uint4*>(cnt);
  for (int l = threadIdx.x; l < rk; l += blockDim.x) cnt4[l] = make_uint4(0, 0, 0, 0);
  const int base = blockIdx.x * kTile + w * kPer;
  int lab[kSteps];
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    const int p = base + i * 32 + lane;
    lab[i] = p < J.f_n ? J.f_label[p] : -1;
  }
  __syncthreads();
  unsigned peers[kSteps];
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    peers[i] = __match_any_sync(0xffffffffu, lab[i]);
    if (lab[i] >= 0 && lane == __ffs(peers[i]) - 1)
      cnt[lab[i] * kScatterWarps + w] += (unsigned short)__popc(peers[i]);
    __syncwarp();
  }
  __syncthreads();
  for (int l = threadIdx.x; l < rk; l += blockDim.x) {
    uint4 c = cnt4[l];
    unsigned run = 0;  // two 16-bit counts per word, in warp order
    unsigned* v = &c.x;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned a = v[q] & 0xffffu, b = v[q] >> 16;
      v[q] = run | ((run + a) << 16);
      run += a + b;
    }
    cnt4[l] = c;
  }
  __syncthreads();
  const int* row = J.hist + (size_t)blockIdx.x * rk;
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    const int l = lab[i];
    int in = 0;
    if (l >= 0) in = cnt[l * kScatterWarps + w];
    __syncwarp();
    if (l >= 0 && lane == __ffs(peers[i]) - 1)
      cnt[l * kScatterWarps + w] = (unsigned short)(in + __popc(peers[i]));
    __syncwarp();
    if (l >= 0) {
      const int p = base + i * 32 + lane;
      const double wt = J.fw[p];
      J.sorted[J.start[l] + row[l] + in + __popc(peers[i] & ((1u << lane) - 1u))] =
          make_double4(rmul(wt, J.fx[p]), rmul(wt, J.fy[p]), rmul(wt, J.fz[p]), wt);
    }
  }
}

// 2^e for a normal power of two.
__device__ __forceinline__ double pow2_bits(int e) {
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// m successive round-to-nearest additions acc <- fl(acc + c), acc >= 0,
// c >= 0, with the exact result of the sequential loop. While acc stays in
// one binade [2^e, 2^(e+1)) every addition adds the same number of ulps
// (c rounded to the ulp grid), unless c's remainder is exactly half an ulp
// (a tie, which depends on acc's parity): those steps, binade crossings and
// accumulators outside [2^-900, 2^900] (where the scaling by the ulp would
// not be exact) are taken one at a time, as is a c that is not >= 0; the rest
// are jumped. One thread runs
// it on the critical path of its cluster, so the scaling is by powers of two
// built from the exponent bits: the library's ilogb and ldexp and two
// divisions per binade took most of the 52 us of a fold with a 5551-point
// zero tail.
__device__ double repeat_add(double acc, double c, long long m) {
  const double two53 = 9007199254740992.0;
  while (m > 0) {
    if (c == 0.0) return radd(acc, 0.0);
    const int e = (int)((__double_as_longlong(acc) >> 52) & 0x7ff) - 1023;
    // (a negative c is no weight, but the caller's to give: it must not jump back)
    if (e < -900 || e > 900 || !(c >= 0.0 && c < pow2_bits(e))) {
      acc = radd(acc, c);
      --m;
      continue;
    }
    const double inv = pow2_bits(52 - e);  // 1 / ulp of acc
    const double cu = c * inv;             // exact: a power of two
    const double q = floor(cu);
    const double r = cu - q;
    if (r == 0.5) {
      acc = radd(acc, c);
      --m;
      continue;
    }
    const double qp = q + (r > 0.5 ? 1.0 : 0.0);  // ulps added per step
    if (qp == 0.0) return acc;  // c rounds away now and at every larger exponent
    const double a = acc * inv;  // integer in [2^52, 2^53)
    const double room = two53 - q - 2.0 - a;
    if (room < 0.0) {
      acc = radd(acc, c);
      --m;
      continue;
    }
    long long k = (long long)floor(room / qp) + 1;
    if (k > m) k = m;
    acc = __dmul_rn(__dadd_rn(a, __dmul_rn((double)k, qp)), pow2_bits(e - 52));  // all exact
    m -= k;
  }
  return acc;
}

// The fold of a cluster: acc <- fl(acc + v) over its members in index order
// (utility.cpp:816-822), one addition after the other, so the largest
// cluster's chain of dependent additions (8.5 cycles each) bounds the kernel.
// Once the sum is large against its members the chain is cut where its result
// is known without it: while acc stays in one binade [2^e, 2^(e+1)), an
// addition of v >= 0 adds RN(v), v rounded to the multiple of acc's ulp u,
// whatever acc is (unless v lies exactly half way between two multiples, where
// acc's parity decides), and sums of such multiples below 2^53 u are exact in
// any order. A warp then takes kFoldBatch members at once: each lane rounds
// its own, and one addition of their exact total finishes the lot if acc
// stays in its binade. A batch with a crossing, a tie, or a member too large
// (or negative by more than the rounding error of a coordinate) is added one
// by one. About one member in n ties and every doubling of n crosses, so below
// kFoldSerial members most batches would fail: those are always added one by
// one. (A prefix sum up to the first such member instead of the one-by-one
// batch took 6000 to 8000 cycles a batch, against 2200.)
constexpr int kFoldRows = 8;
constexpr int kFoldBatch = 32 * kFoldRows;  // members per step
constexpr int kFoldSerial = 1024;           // members always added one by one

// acc + the batch held by the warp (v[j] of lane l is member j * 32 + l, zero
// past the end) where the exact total settles it; false and acc unchanged
// otherwise.
__device__ __forceinline__ bool fold_batch(const double (&v)[kFoldRows], double* acc) {
  const int e = (int)((__double_as_longlong(*acc) >> 52) & 0xfff) - 1023;  // sign in: e > 1023
  if (e < -900 || e > 900) return false;
  const double top = pow2_bits(e - 1);   // larger members would change magic's ulp
  const double neg = -pow2_bits(e - 54);  // a quarter ulp off leaves even the binade's start
  const double half_u = pow2_bits(e - 53), magic = 1.5 * pow2_bits(e);
  double sum = 0.0;
  bool bad = false;
#pragma unroll
  for (int j = 0; j < kFoldRows; ++j) {
    const double q = __dsub_rn(__dadd_rn(magic, v[j]), magic);  // RN(v) to a multiple of u
    bad |= !(v[j] > neg && v[j] < top) || fabs(__dsub_rn(v[j], q)) == half_u;
    sum = __dadd_rn(sum, q);
  }
  if (__any_sync(0xffffffffu, bad)) return false;
  for (int o = 16; o > 0; o >>= 1) sum = __dadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
  const double next = __dadd_rn(*acc, sum);
  if (!(next < pow2_bits(e + 1))) return false;
  *acc = next;
  return true;
}

// acc + the first cnt members of the batch one by one, from the warp's copy in
// shared memory (a broadcast load per member; by shuffles the chain took 40 %
// longer), the next 16 loaded while 16 are added.
__device__ __forceinline__ double fold_serial(const double* comp, int cnt, double acc) {
  double x[16], y[16];
  int e = 0;
  if (cnt >= 16) {
#pragma unroll
    for (int u = 0; u < 16; ++u) x[u] = comp[u];
    for (; e + 32 <= cnt; e += 16) {
#pragma unroll
      for (int u = 0; u < 16; ++u) y[u] = comp[e + 16 + u];
#pragma unroll
      for (int u = 0; u < 16; ++u) acc = radd(acc, x[u]);
#pragma unroll
      for (int u = 0; u < 16; ++u) x[u] = y[u];
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) acc = radd(acc, x[u]);
    e += 16;
  }
  for (; e < cnt; ++e) acc = radd(acc, comp[e]);
  return acc;
}

// Cluster c's centroid (sums / count, utility.cpp:831-841) beside its count, and
// an upper bound on the distance it moved (rounded upward); an empty cluster is
// recorded, and the update compacts (its own entry is not used then).
__device__ __forceinline__ void store_centroid(const double4& s, int c,
                                               const double4* cen, double4* sums, double* shift,
                                               KmState* st) {
  if (!(s.w != 0.0)) {
    sums[c] = s;
    st->any_empty = 1;
    return;
  }
  const double4 o = cen[c];
  const double4 n = make_double4(rdiv(s.x, s.w), rdiv(s.y, s.w), rdiv(s.z, s.w), s.w);
  const double dx = fabs(n.x - o.x), dy = fabs(n.y - o.y), dz = fabs(n.z - o.z);
  const double d2 = __dadd_ru(__dadd_ru(__dmul_ru(dx, dx), __dmul_ru(dy, dy)), __dmul_ru(dz, dz));
  sums[c] = n;
  shift[c] = __dmul_ru(__dsqrt_ru(d2), 1.0 + 1e-13);
}

// One block per cluster, one warp per component (w x, w y, w z, w), each by
// itself: the components reach their crossings and ties at different members,
// and a block that stages the members for all four would wait for the slowest
// in every batch. The next batch is loaded while one is folded. The zero-tail
// points p >= npt are identical copies of grid point 0 (weight w[0],
// coordinates (0, 0, 0)) and come last in their cluster's member list, so
// their part of the fold is a repeated addition of one value (repeat_add).
constexpr int kFoldThreads = 128;

template <int N>
__global__ void __launch_bounds__(kFoldThreads) k_segsum(const __grid_constant__ KmJobs<N> JS) {
  after_previous();
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  KmState* st = J.st;
  if (st->done) return;
  const int n = J.f_n, npt = J.f_npt;
  // the clusters that started as the last points of the list reach over the
  // rest of the box and stay the largest: first come, so that their folds do
  // not start in a second wave of blocks
  const int c = gridDim.x - 1 - blockIdx.x;
  if (c >= st->rk) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* v = reinterpret_cast<const double*>(J.sorted + J.start[c]) + warp;
  int m = J.members[c];
  long long tail = 0;
  if (npt < n && J.f_label[npt] == c) {
    tail = n - npt;
    m -= (int)tail;
  }
  double cur[kFoldRows], nxt[kFoldRows];
  auto load = [&](int q, double (&out)[kFoldRows]) {
#pragma unroll
    for (int j = 0; j < kFoldRows; ++j) {
      const int e = q + j * 32 + lane;
      out[j] = e < m ? v[(size_t)e * 4] : 0.0;
    }
  };
  __shared__ double stage[kFoldThreads / 32][kFoldBatch];
  __shared__ double total[4];
  double* comp = stage[warp];
  double acc = 0.0;
  load(0, nxt);
  for (int q = 0; q < m; q += kFoldBatch) {
#pragma unroll
    for (int j = 0; j < kFoldRows; ++j) cur[j] = nxt[j];
    if (q + kFoldBatch < m) load(q + kFoldBatch, nxt);
    if (q < kFoldSerial || !fold_batch(cur, &acc)) {
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kFoldRows; ++j) comp[j * 32 + lane] = cur[j];
      __syncwarp();
      acc = fold_serial(comp, min(kFoldBatch, m - q), acc);
    }
  }
  if (lane == 0) {
    if (tail) {
      const double w0 = J.fw[npt];
      const double one =
          warp == 3 ? w0 : rmul(w0, warp == 0 ? J.fx[npt] : warp == 1 ? J.fy[npt] : J.fz[npt]);
      acc = repeat_add(acc, one, tail);
    }
    total[warp] = acc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double4 s = make_double4(total[0], total[1], total[2], total[3]);
    if (J.sharded) J.f_sums[c] = s;  // a rank's partial sums
    else store_centroid(s, c, J.cen, J.sums, J.shift, st);
  }
}

// The empty-cluster compaction of utility.cpp:831-853: the loop there fills each
// empty place with the last cluster, again while that one is empty too, and
// shrinks rk. So the clusters below the final rk stay where they are, and the
// k-th empty place (ascending) takes the k-th non-empty cluster from the end.
// One block finds both lists by prefix counts (holes, fillers: scratch of rk
// entries each; sums: the centroids beside their counts); the loop by one thread took 1.8 ms at 3000 centroids.
__device__ int compact_empty(const double4* sums, int rk, double4* cen, int* holes, int* fillers,
                             int* warp_tot) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int per = (rk + 1023) / 1024;
  const int b0 = min(rk, tid * per), b1 = min(rk, b0 + per);
  int mine = 0;
  for (int i = b0; i < b1; ++i) mine += !(sums[i].w != 0.0);
  int inc = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) warp_tot[w] = inc;
  __syncthreads();
  int before = inc - mine, empty = 0;
  for (int q = 0; q < 32; ++q) {
    if (q < w) before += warp_tot[q];
    empty += warp_tot[q];
  }
  const int left = rk - empty;
  for (int i = b0; i < b1; ++i) {
    const double4 s = sums[i];
    if (!(s.w != 0.0)) {
      if (i < left) holes[before] = i;
      ++before;
    } else if (i < left) {
      cen[i] = make_double4(s.x, s.y, s.z, 0.0);
    } else {
      fillers[(rk - 1 - i) - (empty - before)] = i;  // non-empty clusters after i
    }
  }
  __syncthreads();
  // as many fillers at or past `left` as holes below it
  int nholes = 0;
  for (int i = left + tid; i < rk; i += 1024) nholes += sums[i].w != 0.0;
  for (int o = 16; o > 0; o >>= 1) nholes += __shfl_xor_sync(0xffffffffu, nholes, o);
  __syncthreads();
  if (lane == 0) warp_tot[w] = nholes;
  __syncthreads();
  nholes = 0;
  for (int q = 0; q < 32; ++q) nholes += warp_tot[q];
  for (int k = tid; k < nholes; k += 1024) {
    const double4 s = sums[fillers[k]];
    cen[holes[k]] = make_double4(s.x, s.y, s.z, 0.0);
  }
  __syncthreads();
  return left;
}

__device__ __forceinline__ int cell_index(const CellGrid& g, double x, double y, double z) {
  const int nc = g.nc;
  const int ci = min(nc - 1, max(0, (int)floor(x * g.inv_h[0])));
  const int cj = min(nc - 1, max(0, (int)floor(y * g.inv_h[1])));
  const int ck = min(nc - 1, max(0, (int)floor(z * g.inv_h[2])));
  return ci + nc * (cj + nc * ck);
}

// After the folds (whose blocks have done the divisions and the moves), two blocks,
// bound by the latency of their phases, which do not need each other:
//  - block 0 sorts the new centroids (compacted as above where a cluster is empty)
//    into the cell grid (cell_start, cell_cen), the first kCenHeld per thread read
//    once;
//  - block 1 puts them into place and takes the largest move, and for every cell
//    the largest move of a centroid that sat in its 3^3 and 5^3 neighbourhoods
//    before the update (cell_of still holds the previous positions' cells there).
// One block for both took 14.9 us at 2979 centroids, 5.2 at 309.
// update = 0: the cells alone (the first centroids).
constexpr int kCenHeld = 3;

template <int N>
__global__ void __launch_bounds__(1024) k_centroids(const __grid_constant__ KmJobs<N> JS, int update) {
  after_previous();
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  KmState* st = J.st;
  if (st->done) return;
  extern __shared__ unsigned cmax[];  // 4 x ncells + 1 words
  __shared__ int warp_tot[32];
  const CellGrid& g = J.cg;
  const int nc = g.nc, ncells = nc * nc * nc;
  const bool empty = update && st->any_empty;
  if (blockIdx.x == 1) {
    if (!update || empty) return;
    const int rk = st->rk;
    for (int c = threadIdx.x; c < ncells; c += blockDim.x) cmax[c] = 0u;
    __syncthreads();
    // the largest move: one atomic per warp (the moves are >= 0, so their bit
    // patterns order as the values do)
    unsigned long long mx = 0ull;
#pragma unroll kCenHeld
    for (int i = threadIdx.x; i < rk; i += blockDim.x) {
      const double4 c = J.sums[i];
      const double sh = J.shift[i];
      const int was = J.cell_of[i];
      J.cen[i] = make_double4(c.x, c.y, c.z, 0.0);
      J.cell_of[i] = cell_index(g, c.x, c.y, c.z);
      mx = max(mx, (unsigned long long)__double_as_longlong(sh));
      atomicMax(&cmax[was], __float_as_uint(__double2float_ru(sh)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(&st->maxshift_bits, mx);
    __syncthreads();
    // 3^3 and 5^3 neighbourhood maxima together, as separable passes (x, y, z):
    // from one array of cells (or a pair, by radius) into the next pair
    unsigned *a1 = cmax + ncells, *a2 = a1 + ncells, *b2 = a2 + ncells;
    auto pass = [&](int axis, const unsigned* in1, const unsigned* in2, unsigned* out1,
                    unsigned* out2) {
      const int step = axis == 0 ? 1 : axis == 1 ? nc : nc * nc;
      for (int c = threadIdx.x; c < ncells; c += blockDim.x) {
        const int at = (c / step) % nc;
        unsigned m1 = in1[c], m2 = in2[c];
        if (at > 0) {
          m1 = max(m1, in1[c - step]);
          m2 = max(m2, in2[c - step]);
        }
        if (at > 1) m2 = max(m2, in2[c - 2 * step]);
        if (at < nc - 1) {
          m1 = max(m1, in1[c + step]);
          m2 = max(m2, in2[c + step]);
        }
        if (at < nc - 2) m2 = max(m2, in2[c + 2 * step]);
        out1[c] = m1;
        out2[c] = m2;
      }
      __syncthreads();
    };
    pass(0, cmax, cmax, a1, a2);
    pass(1, a1, a2, cmax, b2);
    pass(2, cmax, b2, reinterpret_cast<unsigned*>(J.nbshift),
         reinterpret_cast<unsigned*>(J.nbshift) + kMaxCells);
    return;
  }
  int rk = st->rk;
  const double4* from = J.cen;
  if (empty) {
    // the members' lists of this iteration are done with: scratch
    rk = compact_empty(J.sums, rk, J.cen, J.members, J.start, warp_tot);
    if (threadIdx.x == 0) {
      st->rk = rk;
      st->reset_bounds = 1;
    }
  } else if (update) {
    from = J.sums;
  }
  const bool own_cells = !update || empty;  // else block 1 writes them
  int* sc = reinterpret_cast<int*>(cmax);  // ncells + 1 counters
  for (int c = threadIdx.x; c <= ncells; c += blockDim.x) sc[c] = 0;
  double3 held[kCenHeld];
  int cell[kCenHeld];
#pragma unroll
  for (int q = 0; q < kCenHeld; ++q) {
    const int j = threadIdx.x + q * 1024;
    if (j < rk) {
      const double4 c = from[j];
      held[q] = make_double3(c.x, c.y, c.z);
    }
  }
  __syncthreads();
  auto count = [&](int j, double x, double y, double z) {
    const int id = cell_index(g, x, y, z);
    if (own_cells) J.cell_of[j] = id;
    atomicAdd(&sc[id + 1], 1);
    return id;
  };
#pragma unroll
  for (int q = 0; q < kCenHeld; ++q) {
    const int j = threadIdx.x + q * 1024;
    if (j < rk) cell[q] = count(j, held[q].x, held[q].y, held[q].z);
  }
  for (int j = threadIdx.x + kCenHeld * 1024; j < rk; j += 1024) {
    const double4 c = from[j];
    count(j, c.x, c.y, c.z);
  }
  __syncthreads();
  block_inclusive_scan(sc + 1, ncells, warp_tot);
  for (int c = threadIdx.x; c <= ncells; c += blockDim.x) J.cell_start[c] = sc[c];
  __syncthreads();
  // placement inside a cell is arbitrary: the search compares (d, index) pairs
#pragma unroll
  for (int q = 0; q < kCenHeld; ++q) {
    const int j = threadIdx.x + q * 1024;
    if (j < rk)
      J.cell_cen[atomicAdd(&sc[cell[q]], 1)] =
          make_double4(held[q].x, held[q].y, held[q].z, (double)j);
  }
  for (int j = threadIdx.x + kCenHeld * 1024; j < rk; j += 1024) {
    const double4 c = from[j];
    J.cell_cen[atomicAdd(&sc[cell_index(g, c.x, c.y, c.z)], 1)] =
        make_double4(c.x, c.y, c.z, (double)j);
  }
}

// ---------------------------------------------------------------- final
// Nearest point to every centroid: first minimum over points
// (std::min_element, utility.cpp:926-945). Partial minima per point chunk,
// then an in-order reduction over the chunks.
__global__ void __launch_bounds__(128) k_final_partial(const double* __restrict__ px,
                                                       const double* __restrict__ py,
                                                       const double* __restrict__ pz, int n,
                                                       const double4* __restrict__ cen,
                                                       const KmState* st,
                                                       double* __restrict__ part_d,
                                                       int* __restrict__ part_i) {
  const int rk = st->rk;
  const int j = blockIdx.x * 128 + threadIdx.x;
  const int chunk = blockIdx.y;
  __shared__ double sx[512], sy[512], sz[512];
  double cx = 0, cy = 0, cz = 0;
  if (j < rk) {
    double4 c = cen[j];
    cx = c.x;
    cy = c.y;
    cz = c.z;
  }
  double best = __longlong_as_double(0x7ff0000000000000LL);
  int bi = 0x7fffffff;
  const int base = chunk * kFinalChunk;
  const int end = min(base + kFinalChunk, n);
  for (int p0 = base; p0 < end; p0 += 512) {
    const int m = min(512, end - p0);
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += 128) {
      sx[k] = px[p0 + k];
      sy[k] = py[p0 + k];
      sz[k] = pz[p0 + k];
    }
    __syncthreads();
    for (int k = 0; k < m; ++k) {
      double d1 = rsub(sx[k], cx), d2 = rsub(sy[k], cy), d3 = rsub(sz[k], cz);
      double d = radd(radd(rmul(d1, d1), rmul(d2, d2)), rmul(d3, d3));
      if (d < best) {
        best = d;
        bi = p0 + k;
      }
    }
  }
  if (j < rk) {
    part_d[(size_t)chunk * rk + j] = best;
    part_i[(size_t)chunk * rk + j] = bi;
  }
}

__global__ void k_final_reduce(const double* __restrict__ part_d, const int* __restrict__ part_i,
                               int nchunks, const KmState* st, const int* __restrict__ pidx,
                               int* __restrict__ sel) {
  const int rk = st->rk;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= rk) return;
  double best = __longlong_as_double(0x7ff0000000000000LL);
  int bi = 0;
  for (int c = 0; c < nchunks; ++c) {
    double d = part_d[(size_t)c * rk + j];
    if (d < best) {
      best = d;
      bi = part_i[(size_t)c * rk + j];
    }
  }
  sel[j] = pidx[bi];
}

// The same where the grid gives the points' places, one warp per centroid: the
// kept points of a box of grid points around the centroid, (distance, list
// index) pairs compared, the box doubled until every point outside it (a grid
// spacing or more beyond its faces, less tol) is farther than the nearest found
// or the box is the grid. The zero tail's first point (a copy of grid point 0)
// is compared once. A few points per centroid instead of all of them: 20 us
// against 1.6 ms at 884 736 points and 2979 centroids.
template <int N>
__global__ void __launch_bounds__(128)
    k_final_near(const __grid_constant__ KmJobs<N> JS) {
  const KmJob& J = JS.j[N == 1 ? 0 : blockIdx.y];
  const int rk = J.st->rk;
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j >= rk) return;
  const double4 c = J.cen[j];
  const AssignMap& am = J.am;
  const int n3[3] = {am.nx, am.ny, am.nz};
  const double cc[3] = {c.x, c.y, c.z}, h3[3] = {J.dx[0], J.dx[1], J.dx[2]};
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  double best = inf;
  int bp = 0;
  for (int r = 1;; r *= 2) {
    int lo[3], ext[3];
    double margin = inf;  // every point outside the box is at least this far
    bool all = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double at = floor(cc[d] / h3[d]);
      const int f = (int)fmin(fmax(at, 0.0), (double)(n3[d] - 1));
      lo[d] = max(0, f - r + 1);
      const int hi = min(n3[d] - 1, f + r);
      ext[d] = hi - lo[d] + 1;
      if (lo[d] > 0) {
        margin = fmin(margin, cc[d] - (lo[d] - 1) * h3[d] - J.cg.tol);
        all = false;
      }
      if (hi < n3[d] - 1) {
        margin = fmin(margin, (hi + 1) * h3[d] - cc[d] - J.cg.tol);
        all = false;
      }
    }
    best = inf;
    bp = 0;
    if (am.npt < J.n && lane == 0) {  // the zero tail
      const double d = ref_dist2(J.px[am.npt], J.py[am.npt], J.pz[am.npt], c);
      if (d < best) {
        best = d;
        bp = am.npt;
      }
    }
    const int count = ext[0] * ext[1] * ext[2];
    for (int e = lane; e < count; e += 32) {
      const int ix = lo[0] + e % ext[0], iy = lo[1] + (e / ext[0]) % ext[1],
                iz = lo[2] + e / (ext[0] * ext[1]);
      const int gp = ix + am.nx * (iy + am.ny * iz);
      const int p = am.g2p ? am.g2p[gp] : gp;
      if (p < 0) continue;
      const double d = ref_dist2(J.px[p], J.py[p], J.pz[p], c);
      if (d < best || (d == best && p < bp)) {
        best = d;
        bp = p;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double od = __shfl_xor_sync(0xffffffffu, best, o);
      const int op = __shfl_xor_sync(0xffffffffu, bp, o);
      if (od < best || (od == best && op < bp)) {
        best = od;
        bp = op;
      }
    }
    if (all || (margin > 0.0 && best < margin * margin * (1.0 - 1e-12))) break;
  }
  if (lane == 0) J.sel[j] = J.pidx[bp];
}

// ---------------------------------------------------------------- sharded
// A rank's record per Lloyd iteration: entry 0 carries the labels its last
// assignment changed (.x), entries 1..rk its partial centroid sums.
__global__ void k_shard_header(const KmState* st, double4* __restrict__ send) {
  send[0] = make_double4((double)st->changed, 0.0, 0.0, 0.0);
}

// The loop test of utility.cpp:812 on the ranks' total of changed labels
// (the reference's MPI_Reduce + MPI_Bcast of flag, utility.cpp:908-917),
// then the iteration's resets.
__global__ void k_shard_begin(KmState* st, const double4* __restrict__ recv, int ranks, int stride,
                              double max_f, int max_iter) {
  if (st->done) return;
  if (st->s > 0) {  // n before the first iteration
    long long f = 0;
    for (int q = 0; q < ranks; ++q) f += (long long)recv[(size_t)q * stride].x;
    st->flag = (int)f;
  }
  if (!((double)st->flag > max_f && st->s < max_iter)) {
    st->done = 1;
    return;
  }
  st->s += 1;
  st->changed = 0;
  st->any_empty = 0;
  st->reset_bounds = 0;
  st->maxshift_bits = 0;
}

__device__ __forceinline__ double4 add4(const double4& a, const double4& b) {
  return make_double4(radd(a.x, b.x), radd(a.y, b.y), radd(a.z, b.z), radd(a.w, b.w));
}

// The ranks' partial sums combined in binomial-tree order (at step s = 1, 2,
// 4, ..., rank q takes in rank q + s: the reduce of utility.cpp:825-826 as
// MPICH's binomial algorithm runs it), evaluated rank by rank with a stack of
// completed subtrees: (r0 + r1) + (r2 + r3) for 4 ranks, (r0 + r1) + r2 for 3.
__global__ void k_shard_sums(KmState* st, const double4* __restrict__ recv, int ranks, int stride,
                             const double4* __restrict__ cen, double4* __restrict__ sums,
                             double* __restrict__ shift) {
  if (st->done) return;
  const int rk = st->rk;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= rk) return;
  double4 val[8];
  int lev[8];
  int top = 0;
  for (int q = 0; q < ranks; ++q) {
    double4 v = recv[(size_t)q * stride + 1 + c];
    int l = 0;
    while (top > 0 && lev[top - 1] == l) {
      v = add4(val[top - 1], v);
      --top;
      ++l;
    }
    val[top] = v;
    lev[top] = l;
    ++top;
  }
  double4 acc = val[top - 1];
  for (int i = top - 2; i >= 0; --i) acc = add4(val[i], acc);
  store_centroid(acc, c, cen, sums, shift, st);
}

// One rank's nearest point per centroid: the first minimum over its points
// (findMin, utility.cpp:926-945), as (distance, grid index).
__global__ void k_final_local(const double* __restrict__ part_d, const int* __restrict__ part_i,
                              int nchunks, const KmState* st, const int* __restrict__ pidx,
                              double2* __restrict__ out) {
  const int rk = st->rk;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= rk) return;
  double best = __longlong_as_double(0x7ff0000000000000LL);
  int bi = 0;
  for (int c = 0; c < nchunks; ++c) {
    double d = part_d[(size_t)c * rk + j];
    if (d < best) {
      best = d;
      bi = part_i[(size_t)c * rk + j];
    }
  }
  out[j] = make_double2(best, (double)pidx[bi]);
}

// MPI_MINLOC over the ranks (utility.cpp:946-969): the smallest distance,
// ties to the smaller grid index.
__global__ void k_minloc(const double2* __restrict__ recv, int ranks, int stride,
                         const KmState* st, int* __restrict__ sel) {
  const int rk = st->rk;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= rk) return;
  double2 best = recv[j];
  for (int q = 1; q < ranks; ++q) {
    const double2 v = recv[(size_t)q * stride + j];
    if (v.x < best.x || (v.x == best.x && v.y < best.y)) best = v;
  }
  sel[j] = (int)best.y;
}

// Dynamic shared memory above 48 KB needs an opt-in per kernel and device.
int set_kmeans_smem_attrs() {
  std::lock_guard<std::mutex> attr_lock(attr_mutex());
  static bool done[64] = {};
  int dev = 0;
  ISDF_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && done[dev]) return ISDF_OK;
  ISDF_CUDA(cudaFuncSetAttribute(k_hist<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(int) * kKmeansMaxMu)));
  ISDF_CUDA(cudaFuncSetAttribute(k_scatter<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(short) * kScatterWarps * kKmeansMaxMu)));
  ISDF_CUDA(cudaFuncSetAttribute(k_hist_scan<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(int) * kKmeansMaxMu)));
  // (a batch's histograms, kKmeansBatchMaxMu labels at most, need no opt-in)
  const int cells = (int)(sizeof(unsigned) * (4 * kMaxCells + 1));
  ISDF_CUDA(cudaFuncSetAttribute(k_centroids<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 cells));
  ISDF_CUDA(cudaFuncSetAttribute(k_centroids<kBatchJobs>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, cells));
  if (dev >= 0 && dev < 64) done[dev] = true;
  return ISDF_OK;
}

struct KmBuffers {
  int* pidx;
  double *px, *py, *pz, *pw;
  int* label;
  double4* sorted;  // (w x, w y, w z, w) in cluster order
  int* hist;
  int* members;
  int* start;
  int* tile_cnt;
  double4* cen;
  double4* sums;
  double2* bnd;    // per point (upper, lower) distance bounds
  double* shift;   // per centroid: distance moved in the last update
  int* g2p;        // grid index -> kept-point index
  float* nbshift;  // per cell: largest move of a centroid in its 27-cell neighbourhood
  double* part_d;
  int* part_i;
  KmState* st;
  int* sel;        // behind *st: the two are read back together
  int* cell_start;
  double4* cell_cen;
  int* pcell;        // per point: its cell
  double2* pd12;     // per point: distances to the outside of its 3^3 / 5^3 cell blocks
  int* cell_of;
};

KmBuffers carve(Arena& a, int n, int mu) {
  KmBuffers b;
  const int ntiles = (n + kTile - 1) / kTile;
  const int nfilter = (n + 1023) / 1024;
  const int nchunks = (n + kFinalChunk - 1) / kFinalChunk;
  b.pidx = a.take<int>(n);
  b.px = a.take<double>(n);
  b.py = a.take<double>(n);
  b.pz = a.take<double>(n);
  b.pw = a.take<double>(n);
  b.label = a.take<int>(n);
  b.sorted = a.take<double4>(n);
  b.hist = a.take<int>((size_t)ntiles * mu);
  b.members = a.take<int>(mu);
  b.start = a.take<int>(mu);
  b.tile_cnt = a.take<int>(nfilter);
  b.cen = a.take<double4>(mu);
  b.sums = a.take<double4>(mu);
  b.bnd = a.take<double2>(n);
  b.shift = a.take<double>(mu);
  b.g2p = a.take<int>(n);
  b.nbshift = a.take<float>(2 * (size_t)kMaxCells);  // 3^3 and 5^3 neighbourhoods
  b.part_d = a.take<double>((size_t)nchunks * mu);
  b.part_i = a.take<int>((size_t)nchunks * mu);
  b.st = a.take<KmState>(1 + (sizeof(int) * (size_t)mu + sizeof(KmState) - 1) / sizeof(KmState));
  b.sel = reinterpret_cast<int*>(b.st + 1);
  b.cell_start = a.take<int>((size_t)kMaxCells + 1);
  b.cell_cen = a.take<double4>(mu);
  b.cell_of = a.take<int>(mu);
  b.pcell = a.take<int>(n);
  b.pd12 = a.take<double2>(n);
  return b;
}

// Exchange buffers of a sharded selection.
struct ShardBuffers {
  double4* send;  // (mu + 1): changed count, partial sums
  double4* recv;  // ranks x (mu + 1)
  double2* fsend;  // mu: nearest point per centroid
  double2* frecv;  // ranks x mu
};

ShardBuffers carve_shard(Arena& a, int mu, int ranks) {
  ShardBuffers b;
  b.send = a.take<double4>((size_t)mu + 1);
  b.recv = a.take<double4>((size_t)ranks * (mu + 1));
  b.fsend = a.take<double2>((size_t)mu);
  b.frecv = a.take<double2>((size_t)ranks * mu);
  return b;
}

// The cell grid of the pruned assignment: about 1.5 centroids per cell.
CellGrid cell_grid(const KmeansArgs& args) {
  CellGrid cg;
  const int nc = std::max(1, std::min((int)std::lround(std::cbrt(args.mu / 1.5)), kMaxCellsPerDim));
  cg.nc = nc;
  double lmax = 0.0;
  for (int i = 0; i < 3; ++i) {
    cg.h[i] = args.length[i] / nc;
    cg.inv_h[i] = 1.0 / cg.h[i];
    lmax = std::max(lmax, std::fabs(args.length[i]));
  }
  cg.tol = 1e-9 * lmax;
  return cg;
}

// The job of a whole selection (a sharded one narrows its fold afterwards);
// am: its thread -> point map.
KmJob make_job(const KmeansArgs& args, const KmBuffers& b, const CellGrid& cg,
               const AssignMap& am, int npt) {
  const int n = (int)args.ng;
  KmJob job{};
  job.pidx = b.pidx;
  job.px = b.px;
  job.py = b.py;
  job.pz = b.pz;
  job.label = b.label;
  job.n = n;
  job.sorted = b.sorted;
  job.cen = b.cen;
  job.sums = b.sums;
  job.hist = b.hist;
  job.members = b.members;
  job.start = b.start;
  job.bnd = b.bnd;
  job.shift = b.shift;
  job.nbshift = b.nbshift;
  job.st = b.st;
  job.cell_start = b.cell_start;
  job.cell_cen = b.cell_cen;
  job.cell_of = b.cell_of;
  job.pcell = b.pcell;
  job.pd12 = b.pd12;
  job.cg = cg;
  job.am = am;
  job.f_label = b.label;
  job.fx = b.px;
  job.fy = b.py;
  job.fz = b.pz;
  job.fw = b.pw;
  job.f_n = n;
  job.f_npt = npt;
  job.f_sums = b.sums;
  job.sel = b.sel;
  for (int i = 0; i < 3; ++i) job.dx[i] = args.length[i] / args.num_grid[i];
  job.max_f = 1e-5 * n;  // KmeansTolerance * n (utility.cpp:812)
  job.max_iter = args.max_iter;
  return job;
}

// The map of a whole selection's points (one rank).
AssignMap brick_map(const KmeansArgs& args, int npt) {
  const int n = (int)args.ng;
  AssignMap am{};
  am.nx = args.num_grid[0];
  am.ny = args.num_grid[1];
  am.nz = args.num_grid[2];
  am.nbx = (am.nx + 3) / 4;
  am.nby = (am.ny + 3) / 4;
  am.nbt = (long long)am.nbx * am.nby * ((am.nz + 1) / 2) * 32;
  am.t0 = 0;
  am.npt = npt;
  am.n = n;
  am.p_lo = 0;
  am.p_hi = n;
  am.brick = ((long long)am.nx * am.ny * am.nz == n && am.nbt + n < 0x7fffffffLL);
  am.g2p = nullptr;
  return am;
}

// Grid sizes of the kernels of an iteration: each for the largest of its jobs.
struct LoopDims {
  unsigned jobs = 0, tiles = 0, mu = 0, assign = 0;
  size_t cells_smem = 0;

  void add(const KmJob& job, int mu_, unsigned assign_blocks) {
    ++jobs;
    tiles = std::max(tiles, (unsigned)((job.f_n + kTile - 1) / kTile));
    mu = std::max(mu, (unsigned)mu_);
    assign = std::max(assign, assign_blocks);
    const size_t ncells = (size_t)job.cg.nc * job.cg.nc * job.cg.nc;
    cells_smem = std::max(cells_smem, sizeof(unsigned) * (4 * ncells + 1));
  }
};

// One Lloyd iteration is six launches: the sums, then the centroids and the
// labels. Every kernel returns at once where the loop has stopped.
template <int N>
void launch_sums(const KmJobs<N>& J, const LoopDims& d, const LoopSignal& sig, int* live,
                 LoopQueue& q) {
  const size_t hist_smem = sizeof(int) * (size_t)d.mu;
  const size_t scatter_smem = sizeof(short) * kScatterWarps * (size_t)d.mu;
  launch_early(k_hist<N>, dim3(d.tiles, d.jobs), 256, hist_smem, q, J, sig);
  launch_early(k_hist_scan<N>, dim3((d.mu + 31) / 32, d.jobs), 32 * kScanWarps, hist_smem, q, J, sig,
               live);
  launch_early(k_scatter<N>, dim3(d.tiles, d.jobs), 32 * kScatterWarps, scatter_smem, q, J);
  launch_early(k_segsum<N>, dim3(d.mu, d.jobs), kFoldThreads, 0, q, J);
}

template <int N>
void launch_assign(const KmJobs<N>& J, const LoopDims& d, int update, LoopQueue& q) {
  launch_early(k_centroids<N>, dim3(2, d.jobs), 1024, d.cells_smem, q, J, update);
  launch_early(k_assign_warp<N>, dim3(d.assign, d.jobs), kAssignThreads, 0, q, J, update);
}

// One Lloyd iteration on a queue: a round of the selection's loop.
template <int N>
auto lloyd_round(const KmJobs<N>& J, const LoopDims& d, int* live) {
  return [&J, &d, live](LoopQueue& q, const LoopSignal& sig) {
    launch_sums(J, d, sig, live, q);
    launch_assign(J, d, 1, q);
  };
}

}  // namespace

size_t kmeans_workspace_bytes(long long ng, int mu) {
  Arena a;
  a.counting = true;
  carve(a, (int)ng, mu);
  return a.off;
}

size_t kmeans_shard_workspace_bytes(long long ng, int mu, int ranks) {
  Arena a;
  a.counting = true;
  carve(a, (int)ng, mu);
  carve_shard(a, mu, ranks);
  return a.off;
}

int kmeans_weight(const double* d_psi, long long ng, int nocc, int nv1, int nc1, int nv2, int nc2,
                  double* d_w, cudaStream_t stream) {
  const int same = (nv1 == nv2 && nc1 == nc2);
  unsigned grid = grid_for(ng, 256);
  if (grid > (unsigned)kNumSMs * 16) grid = kNumSMs * 16;
  k_weight<<<grid, 256, 0, stream>>>(d_psi, ng, nocc - nv2, nocc + nc2, nocc - nv1, nocc + nc1,
                                     same, d_w);
  ISDF_CHECK_LAUNCH();
  return ISDF_OK;
}

// libstdc++'s std::random_shuffle(first, last) loop, driven by std::rand(),
// which the reference calls on its npt < mu branch (utility.cpp:679); draw()
// stands in for std::rand().
template <class Draw>
static void shuffle_like_libstdcxx(int* first, int* last, Draw draw) {
  if (first == last) return;
  for (int* i = first + 1; i != last; ++i) {
    int* j = first + draw() % ((i - first) + 1);
    if (i != j) std::swap(*i, *j);
  }
}
static void shuffle_like_libstdcxx(int* first, int* last) {
  shuffle_like_libstdcxx(first, last, [] { return std::rand(); });
}

// The sequence std::rand() gives after std::srand(seed), from glibc's own
// generator on a private state (initstate_r / random_r, the generator behind
// rand()), so that ranks sharing one process do not share their draws.
struct SeededRand {
  random_data data;
  char state[128];
  explicit SeededRand(unsigned seed) {
    std::memset(&data, 0, sizeof(data));
    std::memset(state, 0, sizeof(state));
    initstate_r(seed, state, sizeof(state), &data);
  }
  int operator()() {
    int32_t r = 0;
    random_r(&data, &r);
    return (int)r;
  }
};

// piv = [distinct selected points ascending | the rest ascending]
// (unique, utility.cpp:617-629, and utility.cpp:973-983); returns rk_eff. The
// rest is written gap by gap between the selected points.
static int piv_from_selection(std::vector<int>& sel, int n, int* piv) {
  std::sort(sel.begin(), sel.end());
  sel.erase(std::unique(sel.begin(), sel.end()), sel.end());
  const int rk_eff = (int)sel.size();
  std::copy(sel.begin(), sel.end(), piv);
  int* out = piv + rk_eff;
  int from = 0;
  for (int k = 0; k <= rk_eff; ++k) {
    const int to = k < rk_eff ? sel[k] : n;
    for (int i = from; i < to; ++i) *out++ = i;
    from = to + 1;
  }
  return rk_eff;
}

int kmeans_select(const KmeansArgs& args, Arena& arena, cudaStream_t stream, KmeansResult* res,
                  Transport* shard) {
  const int n = (int)args.ng;
  const int mu = args.mu;
  if (n <= 0 || mu <= 0 || mu > kKmeansMaxMu) return record_error(ISDF_ERR_ARG, "kmeans: bad n/mu");
  if (args.ng > 0x7fffffffLL) return record_error(ISDF_ERR_UNSUPPORTED, "kmeans: Ng >= 2^31");
  const int ranks = shard ? shard->size : 1;
  if (ranks > kKmeansMaxRanks || ranks > n)
    return record_error(ISDF_ERR_UNSUPPORTED, "kmeans: more ranks than supported or points");
  KmBuffers b = carve(arena, n, mu);
  ShardBuffers sb{};
  if (shard) sb = carve_shard(arena, mu, ranks);
  if (arena.overflowed()) return record_error(ISDF_ERR_NOMEM, "kmeans: workspace too small");
  // this rank's points of the n-long list (utility.cpp:682-689); all of them at one rank
  const int lo = shard ? (int)block_start(n, ranks, shard->rank) : 0;
  const int cnt = shard ? (int)block_count(n, ranks, shard->rank) : n;
  const int nfilter = (n + 1023) / 1024;
  const int nchunks = (n + kFinalChunk - 1) / kFinalChunk;
  // a rank of a sharded selection draws from its own generator (below)
  if (args.rand_seed >= 0 && !shard) std::srand((unsigned)args.rand_seed);
  // warm start: the caller's previous pivots, read before piv is rewritten
  std::vector<int> prev;
  if (args.warm && n > 1 && args.piv[0] != args.piv[1]) {
    prev.assign(args.piv, args.piv + mu);
    for (int v : prev)
      if (v < 0 || v >= n) return record_error(ISDF_ERR_ARG, "kmeans: warm-start pivot outside the grid");
  }
  res->warm_pivots = -1;

  // filter: maxW, kept-point compaction, zero tail
  ISDF_CUDA(cudaMemsetAsync(b.st, 0, sizeof(KmState), stream));
  ISDF_CUDA(cudaMemsetAsync(b.pidx, 0, sizeof(int) * (size_t)n, stream));
  k_maxw<<<kNumSMs * 4, 256, 0, stream>>>(args.d_w, n, b.st);
  k_filter_count<<<nfilter, 256, 0, stream>>>(args.d_w, n, b.st, b.tile_cnt);
  k_scan_small<<<1, 1024, 0, stream>>>(b.tile_cnt, nfilter, &b.st->npt);
  k_filter_scatter<<<nfilter, 256, 0, stream>>>(args.d_w, n, b.st, b.tile_cnt, b.pidx);
  ISDF_CHECK_LAUNCH();
  KmState hst;
  ISDF_TRY(read_back(&hst, b.st, sizeof(KmState), stream));
  const int npt = hst.npt;
  res->npt = npt;

  if (npt < mu) {
    // utility.cpp:667-681: piv from the kept list, then a shuffled tail.
    std::memset(args.piv, 0, sizeof(int) * (size_t)n);
    std::vector<int> index(n, 0);
    ISDF_TRY(read_back(index.data(), b.pidx, sizeof(int) * (size_t)npt, stream));
    int k0 = 0, k1 = 0;
    for (int i = 0; i < npt; i++) {
      if (i == index[k0]) {
        args.piv[k0] = i;
        k0 = std::min(k0 + 1, mu - 1);
      } else {
        args.piv[npt + k1] = i;
        k1++;
      }
    }
    if (shard) {
      // every rank process of the reference starts from libc's initial
      // state (seed 1) unless the caller seeds it
      SeededRand draw(args.rand_seed >= 0 ? (unsigned)args.rand_seed : 1u);
      shuffle_like_libstdcxx(args.piv + npt, args.piv + n, [&] { return draw(); });
    } else {
      shuffle_like_libstdcxx(args.piv + npt, args.piv + n);
    }
    res->rk_eff = mu;
    res->iters = -1;
    res->launches = 4 + (readback_mailbox() ? 2 : 0);
    return ISDF_OK;
  }

  const double dx0 = args.length[0] / args.num_grid[0];
  const double dx1 = args.length[1] / args.num_grid[1];
  const double dx2 = args.length[2] / args.num_grid[2];
  std::vector<int> cinit;
  if (!prev.empty()) {
    // utility.cpp:725-749: the previous pivots whose weight passes the
    // filter, in their order, then the first kept points not among them
    // (at most mu kept points are examined: each one either joins or is
    // one of the kept previous pivots)
    ISDF_CUDA(cudaMemcpyAsync(b.sel, prev.data(), sizeof(int) * (size_t)mu,
                              cudaMemcpyHostToDevice, stream));
    k_gather_w<<<grid_for(mu, 256), 256, 0, stream>>>(args.d_w, b.sel, mu, b.part_d);
    ISDF_CHECK_LAUNCH();
    std::vector<double> wprev(mu);
    std::vector<int> head(mu);
    ISDF_TRY(read_back(wprev.data(), b.part_d, sizeof(double) * (size_t)mu, stream));
    ISDF_TRY(read_back(head.data(), b.pidx, sizeof(int) * (size_t)mu, stream));
    double maxw;
    std::memcpy(&maxw, &hst.maxw_bits, sizeof(double));
    const double thr = 1e-8 * maxw;
    cinit.reserve(mu);
    for (int i = 0; i < mu; ++i)
      if (wprev[i] > thr) cinit.push_back(prev[i]);
    res->warm_pivots = (int)cinit.size();
    std::vector<char> in((size_t)n, 0);
    for (int c : cinit) in[c] = 1;
    for (int k = 0; (int)cinit.size() < mu && k < mu; ++k)
      if (!in[head[k]]) cinit.push_back(head[k]);
    ISDF_CUDA(cudaMemcpyAsync(b.sel, cinit.data(), sizeof(int) * (size_t)mu,
                              cudaMemcpyHostToDevice, stream));
  }
  k_points<<<grid_for(n, 256), 256, 0, stream>>>(b.pidx, args.d_w, n, args.num_grid[0],
                                                 args.num_grid[1], dx0, dx1, dx2, b.px, b.py,
                                                 b.pz, b.pw, mu, b.cen);
  if (!prev.empty())
    k_warm_centroids<<<grid_for(mu, 256), 256, 0, stream>>>(b.sel, mu, args.num_grid[0],
                                                            args.num_grid[1], dx0, dx1, dx2,
                                                            b.cen);
  {
    KmState init{};
    init.flag = n;
    init.changed = n;
    init.rk = mu;
    init.npt = npt;
    init.maxw_bits = hst.maxw_bits;
    ISDF_CUDA(cudaMemcpyAsync(b.st, &init, sizeof(KmState), cudaMemcpyHostToDevice, stream));
  }
  const CellGrid cg = cell_grid(args);
  AssignMap am = brick_map(args, npt);
  am.p_lo = lo;
  am.p_hi = lo + cnt;
  if (am.brick && npt < n) {
    ISDF_CUDA(cudaMemsetAsync(b.g2p, 0xff, sizeof(int) * (size_t)n, stream));
    k_grid_to_point<<<grid_for(npt, 256), 256, 0, stream>>>(b.pidx, npt, b.g2p);
    am.g2p = b.g2p;
  }
  const int kept_hi = std::min(lo + cnt, npt);  // this rank's kept points: [lo, kept_hi)
  const int tail_loc = std::max(0, lo + cnt - std::max(npt, lo));
  if (am.brick && shard) {
    // the bricks of the z planes that hold this rank's kept points
    if (lo < kept_hi) {
      int ends[2];
      ISDF_TRY(read_back(&ends[0], b.pidx + lo, sizeof(int), stream));
      ISDF_TRY(read_back(&ends[1], b.pidx + kept_hi - 1, sizeof(int), stream));
      const long long plane = (long long)am.nx * am.ny;
      const long long bz0 = ends[0] / plane / 2, bz1 = ends[1] / plane / 2;
      const long long per_bz = (long long)am.nbx * am.nby * 32;
      am.t0 = bz0 * per_bz;
      am.nbt = (bz1 - bz0 + 1) * per_bz;
    } else {
      am.nbt = 0;
    }
  }
  const unsigned pgrid = am.brick ? grid_for(am.nbt + tail_loc, kAssignThreads)
                                  : grid_for(cnt, kAssignThreads);
  k_point_cells<<<grid_for(n, 256), 256, 0, stream>>>(b.px, b.py, b.pz, n, cg, b.pcell, b.pd12);
  KmJobs<1> jobs;
  KmJob& job = jobs.j[0];
  job = make_job(args, b, cg, am, npt);
  if (shard) {
    job.f_label += lo;
    job.fx += lo;
    job.fy += lo;
    job.fz += lo;
    job.fw += lo;
    job.f_n = cnt;
    job.f_npt = std::max(0, std::min(npt - lo, cnt));
    job.f_sums = sb.send + 1;
    job.sharded = 1;
  }
  LoopDims dims;
  dims.add(job, mu, pgrid);
  ISDF_TRY(set_kmeans_smem_attrs());
  LoopQueue queue(stream);
  launch_assign(jobs, dims, 0, queue);
  ISDF_CHECK_LAUNCH();
  // Sharded: the rank folds its own points [lo, lo + cnt) (utility.cpp:813-822),
  // the ranks exchange their partial sums and changed-label counts (one
  // all-gather per iteration, utility.cpp:825-826,908-917), and every rank
  // combines them in the same order, so that all ranks hold the same
  // centroids without a broadcast. Its collectives keep its iterations out of
  // the loop's graphs.
  const size_t rec_bytes = sizeof(double4) * ((size_t)mu + 1);
  std::vector<size_t> rcounts(ranks, rec_bytes), rdispls(ranks);
  for (int q = 0; q < ranks; ++q) rdispls[q] = (size_t)q * rec_bytes;
  const LoopSignal no_signal{nullptr};
  auto launch_chunk = [&]() -> int {
    for (int it = 0; it < kIterChunk; ++it) {
      launch_sums(jobs, dims, no_signal, nullptr, queue);
      k_shard_header<<<1, 1, 0, stream>>>(b.st, sb.send);
      ISDF_CHECK_LAUNCH();
      ISDF_TRY(shard->allgatherv(sb.send, rec_bytes, sb.recv, rcounts.data(), rdispls.data(),
                                 stream));
      k_shard_begin<<<1, 1, 0, stream>>>(b.st, sb.recv, ranks, mu + 1, job.max_f,
                                         args.max_iter);
      k_shard_sums<<<grid_for(mu, 128), 128, 0, stream>>>(b.st, sb.recv, ranks, mu + 1, b.cen,
                                                          b.sums, b.shift);
      launch_assign(jobs, dims, 1, queue);
      ISDF_CHECK_LAUNCH();
    }
    return ISDF_OK;
  };
  int chunks = 0;
  const int max_chunks = args.max_iter / kIterChunk + 2;
  std::optional<Loop> loop;  // (taken apart once the selection has been read back)
  if (!shard) {
    loop.emplace(stream);
    const auto round = lloyd_round(jobs, dims, nullptr);
    ISDF_TRY(loop->start(kAheadIters, round));
    // the caller's piv is paged in while the loop runs
    std::memset(args.piv, 0, sizeof(int) * (size_t)n);
    ISDF_TRY(loop->finish((long long)args.max_iter + 1, kBodyIters, kSlackIters, round,
                          [&](bool* over) -> int {
                            ISDF_TRY(read_back(&hst, b.st, sizeof(KmState), stream));
                            *over = hst.done != 0;
                            return ISDF_OK;
                          }));
  } else {
    std::memset(args.piv, 0, sizeof(int) * (size_t)n);
    for (;;) {
      ISDF_TRY(launch_chunk());
      ISDF_TRY(read_back(&hst, b.st, sizeof(KmState), stream));
      if (hst.done) break;
      if (++chunks > max_chunks) return record_error(ISDF_ERR_CUDA, "kmeans: loop did not stop");
    }
  }

  // the nearest point to every centroid
  if (!shard && am.brick) {
    k_final_near<1><<<grid_for(mu, 4), 128, 0, stream>>>(jobs);
  } else if (!shard) {
    dim3 fgrid((unsigned)((mu + 127) / 128), (unsigned)nchunks);
    k_final_partial<<<fgrid, 128, 0, stream>>>(b.px, b.py, b.pz, n, b.cen, b.st, b.part_d,
                                               b.part_i);
    k_final_reduce<<<grid_for(mu, 128), 128, 0, stream>>>(b.part_d, b.part_i, nchunks, b.st,
                                                          b.pidx, b.sel);
  } else {
    // each rank's first minimum over its points, then MINLOC over the ranks
    const int rk = hst.rk;
    const int nch = (cnt + kFinalChunk - 1) / kFinalChunk;
    dim3 fgrid((unsigned)((rk + 127) / 128), (unsigned)nch);
    k_final_partial<<<fgrid, 128, 0, stream>>>(b.px + lo, b.py + lo, b.pz + lo, cnt, b.cen, b.st,
                                               b.part_d, b.part_i);
    k_final_local<<<grid_for(rk, 128), 128, 0, stream>>>(b.part_d, b.part_i, nch, b.st,
                                                         b.pidx + lo, sb.fsend);
    ISDF_CHECK_LAUNCH();
    const size_t fb = sizeof(double2) * (size_t)mu;
    std::vector<size_t> fc(ranks, fb), fd(ranks);
    for (int q = 0; q < ranks; ++q) fd[q] = (size_t)q * fb;
    ISDF_TRY(shard->allgatherv(sb.fsend, fb, sb.frecv, fc.data(), fd.data(), stream));
    k_minloc<<<grid_for(rk, 128), 128, 0, stream>>>(sb.frecv, ranks, mu, b.st, b.sel);
  }
  ISDF_CHECK_LAUNCH();
  std::vector<char> out(sizeof(KmState) + sizeof(int) * (size_t)mu);
  ISDF_TRY(read_back(out.data(), b.st, out.size(), stream));
  std::memcpy(&hst, out.data(), sizeof(KmState));
  if (!hst.done) return record_error(ISDF_ERR_CUDA, "kmeans: loop did not stop");
  std::vector<int> sel(hst.rk);
  std::memcpy(sel.data(), out.data() + sizeof(KmState), sizeof(int) * sel.size());
  res->rk_eff = piv_from_selection(sel, n, args.piv);
  res->iters = hst.s;
  res->search_frac = (double)hst.searches / ((double)cnt * (hst.s + 1));
  // filter, points, cells, first assignment, the loop's rounds, the final
  // search, and the reads through the mapped mailbox
  res->launches = 4 + 4 + (am.g2p ? 1 : 0) + hst.rounds * (shard ? 9 : 6) + (am.brick && !shard ? 1 : 2) +
                  (readback_mailbox() ? chunks + 2 : 0);
  return ISDF_OK;
}

// ===================================================================== batched small selections
// Several small K-means selections at once (the serving loop's batches of small
// requests): the kernels of kmeans_select with a job per blockIdx.y, up to
// kBatchJobs of them, in one loop that ends when the last job has. A
// small selection alone is bound by the latency of its launches, so a batch
// costs little more than one; piv is the single selection's bit for bit, the
// kernels being the same. Eight 36^3 systems with 256 centroids: 28.0 ms in one
// cooperative launch of a group of CTAs per system (brute-force assignment,
// group barriers between the phases), 6.9 ms here.
namespace {

// The states and selections of a batch lie in one block, so that one copy
// initialises them and one reads them back.
constexpr size_t kBatchRecord = sizeof(KmState) + sizeof(int) * kKmeansBatchMaxMu;

int select_group(const KmeansArgs* args, int count, Arena& arena, cudaStream_t stream,
                 KmeansResult* res) {
  std::vector<KmBuffers> bufs(count);
  char* records = arena.take<char>(kBatchRecord * (size_t)count);
  int* live = arena.take<int>(1);
  for (int r = 0; r < count; ++r) {
    bufs[r] = carve(arena, (int)args[r].ng, args[r].mu);
    bufs[r].st = reinterpret_cast<KmState*>(records + kBatchRecord * (size_t)r);
    bufs[r].sel = reinterpret_cast<int*>(bufs[r].st + 1);
  }
  if (arena.overflowed()) return record_error(ISDF_ERR_NOMEM, "kmeans batch: workspace too small");
  // filter: maxW, kept-point compaction, zero tail (per request)
  ISDF_CUDA(cudaMemsetAsync(records, 0, kBatchRecord * (size_t)count, stream));
  for (int r = 0; r < count; ++r) {
    const int n = (int)args[r].ng;
    const int nfilter = (n + 1023) / 1024;
    const KmBuffers& b = bufs[r];
    ISDF_CUDA(cudaMemsetAsync(b.pidx, 0, sizeof(int) * (size_t)n, stream));
    k_maxw<<<kNumSMs * 4, 256, 0, stream>>>(args[r].d_w, n, b.st);
    k_filter_count<<<nfilter, 256, 0, stream>>>(args[r].d_w, n, b.st, b.tile_cnt);
    k_scan_small<<<1, 1024, 0, stream>>>(b.tile_cnt, nfilter, &b.st->npt);
    k_filter_scatter<<<nfilter, 256, 0, stream>>>(args[r].d_w, n, b.st, b.tile_cnt, b.pidx);
  }
  ISDF_CHECK_LAUNCH();
  std::vector<char> host(kBatchRecord * (size_t)count);
  ISDF_TRY(read_back(host.data(), records, host.size(), stream));
  auto state = [&](int r) -> KmState {
    KmState st;
    std::memcpy(&st, host.data() + kBatchRecord * (size_t)r, sizeof(st));
    return st;
  };
  KmJobs<kBatchJobs> jobs;
  LoopDims dims;
  int max_iter = 0;
  std::vector<int> slot;  // request of each job
  for (int r = 0; r < count; ++r) {
    const KmeansArgs& a = args[r];
    const int n = (int)a.ng, mu = a.mu;
    const KmBuffers& b = bufs[r];
    const KmState hst = state(r);
    res[r] = KmeansResult();
    res[r].npt = hst.npt;
    if (a.rand_seed >= 0) std::srand((unsigned)a.rand_seed);
    if (hst.npt < mu) {
      // utility.cpp:667-681: piv from the kept list, then a shuffled tail
      std::memset(a.piv, 0, sizeof(int) * (size_t)n);
      std::vector<int> index(n, 0);
      ISDF_TRY(read_back(index.data(), b.pidx, sizeof(int) * (size_t)hst.npt, stream));
      int k0 = 0, k1 = 0;
      for (int i = 0; i < hst.npt; i++) {
        if (i == index[k0]) {
          a.piv[k0] = i;
          k0 = std::min(k0 + 1, mu - 1);
        } else {
          a.piv[hst.npt + k1] = i;
          k1++;
        }
      }
      shuffle_like_libstdcxx(a.piv + hst.npt, a.piv + n);
      res[r].rk_eff = mu;
      res[r].iters = -1;
      continue;
    }
    const double dx0 = a.length[0] / a.num_grid[0];
    const double dx1 = a.length[1] / a.num_grid[1];
    const double dx2 = a.length[2] / a.num_grid[2];
    k_points<<<grid_for(n, 256), 256, 0, stream>>>(b.pidx, a.d_w, n, a.num_grid[0], a.num_grid[1],
                                                   dx0, dx1, dx2, b.px, b.py, b.pz, b.pw, mu,
                                                   b.cen);
    const CellGrid cg = cell_grid(a);
    AssignMap am = brick_map(a, hst.npt);
    if (hst.npt < n) {
      ISDF_CUDA(cudaMemsetAsync(b.g2p, 0xff, sizeof(int) * (size_t)n, stream));
      k_grid_to_point<<<grid_for(hst.npt, 256), 256, 0, stream>>>(b.pidx, hst.npt, b.g2p);
      am.g2p = b.g2p;
    }
    k_point_cells<<<grid_for(n, 256), 256, 0, stream>>>(b.px, b.py, b.pz, n, cg, b.pcell, b.pd12);
    KmState init{};
    init.flag = n;
    init.changed = n;
    init.rk = mu;
    init.npt = hst.npt;
    init.maxw_bits = hst.maxw_bits;
    std::memcpy(host.data() + kBatchRecord * (size_t)r, &init, sizeof(init));
    KmJob& job = jobs.j[slot.size()];
    job = make_job(a, b, cg, am, hst.npt);
    dims.add(job, mu, grid_for(am.nbt + (n - hst.npt), kAssignThreads));
    max_iter = std::max(max_iter, a.max_iter);
    slot.push_back(r);
  }
  ISDF_CHECK_LAUNCH();
  if (slot.empty()) return ISDF_OK;
  const int nj = (int)slot.size();
  ISDF_CUDA(cudaMemcpyAsync(records, host.data(), host.size(), cudaMemcpyHostToDevice, stream));
  ISDF_CUDA(cudaMemcpyAsync(live, &nj, sizeof(int), cudaMemcpyHostToDevice, stream));
  ISDF_TRY(set_kmeans_smem_attrs());
  LoopQueue queue(stream);
  launch_assign(jobs, dims, 0, queue);
  ISDF_CHECK_LAUNCH();
  Loop loop(stream);
  const auto round = lloyd_round(jobs, dims, live);
  ISDF_TRY(loop.start(kAheadIters, round));
  ISDF_TRY(loop.finish((long long)max_iter + 1, kBodyIters, kSlackIters, round,
                       [&](bool* over) -> int {
                         int left = 0;
                         ISDF_TRY(read_back(&left, live, sizeof(int), stream));
                         *over = left <= 0;
                         return ISDF_OK;
                       }));
  k_final_near<kBatchJobs><<<dim3(grid_for(dims.mu, 4), dims.jobs), 128, 0, stream>>>(jobs);
  ISDF_CHECK_LAUNCH();
  ISDF_TRY(read_back(host.data(), records, host.size(), stream));
  for (int r : slot) {
    const KmState hst = state(r);
    if (!hst.done) return record_error(ISDF_ERR_CUDA, "kmeans batch: loop did not stop");
    std::vector<int> sel(hst.rk);
    std::memcpy(sel.data(), host.data() + kBatchRecord * (size_t)r + sizeof(KmState),
                sizeof(int) * sel.size());
    res[r].iters = hst.s;
    res[r].search_frac = (double)hst.searches / ((double)args[r].ng * (hst.s + 1));
    res[r].rk_eff = piv_from_selection(sel, (int)args[r].ng, args[r].piv);
    res[r].launches = 8 + hst.rounds * 6 / nj;
  }
  return ISDF_OK;
}

}  // namespace

size_t kmeans_batch_workspace_bytes(long long ng, int mu) {
  Arena a;
  a.counting = true;
  a.take<char>(kBatchRecord);
  a.take<int>(1);
  carve(a, (int)ng, mu);
  return a.off;
}

int kmeans_select_batch(const KmeansArgs* args, int count, Arena& arena, cudaStream_t stream,
                        KmeansResult* res) {
  for (int r = 0; r < count; ++r) {
    const KmeansArgs& a = args[r];
    if (a.ng <= 1 || a.ng > kKmeansBatchMaxNg || a.mu <= 0 || a.mu > kKmeansBatchMaxMu ||
        a.mu > a.ng || a.max_iter < 0 || a.warm)
      return record_error(ISDF_ERR_UNSUPPORTED, "kmeans batch: request outside the batched sizes");
  }
  // a group's buffers are free once its results have been read back
  const size_t mark = arena.off;
  for (int r = 0; r < count; r += kBatchJobs) {
    arena.off = mark;
    ISDF_TRY(select_group(args + r, std::min(kBatchJobs, count - r), arena, stream, res + r));
  }
  return ISDF_OK;
}

}  // namespace isdf_b200
