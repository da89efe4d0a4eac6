// QRCP interpolation-point selection on sm_100a.
//
// Reference: src/cpu/getpoints_QRCP.cpp:11-500 (CPU only; the reference's GPU
// entry point has no selector). Same algorithm:
//   numPre = IRound(sqrt(mu * f)), f = 1.5 in the reference   (:82-86)
//   G1, G2 = srand48(seed) Gaussian draws, orthonormal columns (:143-189)
//   A = psi_S1 G1, B = psi_S2 G2 (Ng x numPre)                (:201-207)
//   MG(i + j*numPre, r) = B(r, i) A(r, j); column norms        (:228-235)
//   keep columns with norm^2 > 1e-5 * max                      (:272-284)
//   column-pivoted QR of the kept columns; piv = MGIdx[pivots] (:440-457)
//
// B200 form. MG (numPre^2 x Ng: 19.5 GB at Si64 with f = 2.5) is never
// stored. Column-pivoted Householder QR picks, at every step, the column with
// the largest residual norm; that is the same sequence as pivoted Gram-Schmidt
// on the columns x_r = vec(B_r (x) A_r). Step k:
//   * pick the first column (in the current pivoted order) of maximal
//     residual norm, swap positions as the LAPACK routine does;
//   * q_k = x_pk orthogonalised against q_0..q_{k-1} (two passes), normalised;
//   * every residual norm is downdated with t_r = q_k . x_r, which is
//     t_r = sum_j A(r, j) (B_r Qm)_j, Qm(i, j) = q_k[i + j*numPre]: one
//     FP64 tensor-core tile GEMM over all columns with the row dot fused into
//     its epilogue, and the multiplicative downdate of LAPACK's dgeqpf,
//     nu <- nu sqrt(max(0, 1 - (t/nu)^2));
//   * where dgeqpf's cancellation test fires (LAPACK Working Note 176:
//     temp (nu / nu_ref)^2 <= sqrt(eps), eps = 2^-53), the downdated value is
//     not used: dgeqpf then recomputes the norm of the column's transformed
//     trailing part, i.e. of its residual after the k+1 projections; here
//     that residual is formed from the column's features (projected on
//     q_0..q_k twice) and its norm becomes both nu and the new reference nu_ref.
// Orthonormalising G by Householder QR instead of the reference's dgesvd
// changes G1, G2 by orthogonal factors: MG changes by an orthogonal matrix on
// its left, which leaves the column norms and the pivot sequence unchanged.
#include <mutex>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "arena.h"
#include "common.cuh"
#include "dgemm.cuh"
#include "fit.h"
#include "loop_graph.h"
#include "readback.h"
#include "qrcp.h"
#include "solve.h"

namespace isdf_b200 {

namespace {

constexpr int kMaxPre = 128;  // numPre limit: one 128-wide tile holds every column of Qm
constexpr int kRecomputeGrid = 148;

struct QrState {
  unsigned long long maxbits;  // max norm of the columns before the filter (bit pattern)
  int done;
  int nrec;                    // columns flagged for a norm recompute in this step
  int ntot;
  int total_rec;               // norms recomputed over the whole selection
  int k;                       // pivots picked
  int step;                    // the running step (k - 1), -1 where there is none
  int rounds;                  // steps begun, with or without a pivot
  int pad;
};

// The columns whose residual norm is the largest, by block of a pivot step's last
// kernels: the largest norm and the first position (in the pivoted order) holding
// it, as LAPACK's idamax over the remaining columns picks it.
struct Best {
  double nu;
  int pos;
};

__device__ __forceinline__ Best better(const Best& a, const Best& b) {
  return a.nu > b.nu || (a.nu == b.nu && a.pos < b.pos) ? a : b;
}

__device__ __forceinline__ Best warp_best(Best v) {
  for (int o = 16; o > 0; o >>= 1) {
    Best u;
    u.nu = __shfl_xor_sync(0xffffffffu, v.nu, o);
    u.pos = __shfl_xor_sync(0xffffffffu, v.pos, o);
    v = better(v, u);
  }
  return v;
}

// dgeqpf's recompute threshold sqrt(eps), eps = dlamch('Epsilon') = 2^-53.
__device__ __forceinline__ double tol3z() { return sqrt(1.1102230246251565e-16); }

// The downdate of one active column's residual norm with t = q_k . x_c, as
// dgeqpf does it. Returns false (and lists the column) where the cancellation
// test fires: that column's norm is recomputed exactly after this kernel.
__device__ __forceinline__ bool downdate_norm(int c, double t, double* nu, const double* nu0,
                                              QrState* st, int* rec_list) {
  const double v = nu[c];
  if (v == 0.0) return true;
  const double ratio = fabs(t) / v;
  const double temp = fmax(1.0 - ratio * ratio, 0.0);
  const double rel = v / nu0[c];
  if (temp * rel * rel <= tol3z()) {
    rec_list[atomicAdd(&st->nrec, 1)] = c;
    return false;
  }
  nu[c] = v * sqrt(temp);
  return true;
}

// ------------------------------------------------------------- norms, filter
// Squared MG column norm per grid point, summed j-outer, i-inner with
// explicit rounding as the reference's loop (getpoints_QRCP.cpp:228-235).
__global__ void k_mg_norm(const double* __restrict__ A, const double* __restrict__ B, long long n,
                          int p, double* __restrict__ norm2, QrState* st) {
  double mx = 0.0;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < p; ++j) {
      const double a = A[r + (long long)j * n];
      for (int i = 0; i < p; ++i) {
        const double mg = rmul(B[r + (long long)i * n], a);
        s = radd(s, rmul(mg, mg));
      }
    }
    norm2[r] = s;
    mx = fmax(mx, s);
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx > 0.0)
    atomicMax(&st->maxbits, (unsigned long long)__double_as_longlong(mx));
}

__global__ void __launch_bounds__(256) k_keep_count(const double* __restrict__ norm2, long long n,
                                                    const QrState* st, int* tile_cnt) {
  const double thr = rmul(__longlong_as_double((long long)st->maxbits), 1e-5);
  __shared__ int wc[8];
  const long long base = (long long)blockIdx.x * 1024;
  int c = 0;
  for (int k = 0; k < 4; ++k) {
    const long long i = base + k * 256 + threadIdx.x;
    if (i < n && norm2[i] > thr) ++c;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) wc[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < 8; ++w) t += wc[w];
    tile_cnt[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(1024) k_scan_tiles(int* cnt, int ntiles, int* total) {
  __shared__ int part[1024];
  const int per = (ntiles + 1023) / 1024;
  const int lo = threadIdx.x * per, hi = min(lo + per, ntiles);
  int s = 0;
  for (int i = lo; i < hi; ++i) s += cnt[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int run = threadIdx.x ? part[threadIdx.x - 1] : 0;
  for (int i = lo; i < hi; ++i) {
    const int v = cnt[i];
    cnt[i] = run;
    run += v;
  }
  if (threadIdx.x == 1023) *total = part[1023];
}

__global__ void __launch_bounds__(256) k_keep_scatter(const double* __restrict__ norm2, long long n,
                                                      const QrState* st, const int* tile_off,
                                                      int* __restrict__ idx) {
  const double thr = rmul(__longlong_as_double((long long)st->maxbits), 1e-5);
  __shared__ int wc[8][4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long base = (long long)blockIdx.x * 1024;
  unsigned bal[4];
  for (int k = 0; k < 4; ++k) {
    const long long i = base + k * 256 + threadIdx.x;
    bal[k] = __ballot_sync(0xffffffffu, i < n && norm2[i] > thr);
    if (lane == 0) wc[wid][k] = __popc(bal[k]);
  }
  __syncthreads();
  const int off = tile_off[blockIdx.x];
  for (int k = 0; k < 4; ++k) {
    int before = 0;
    for (int kk = 0; kk < k; ++kk)
      for (int w = 0; w < 8; ++w) before += wc[w][kk];
    for (int w = 0; w < wid; ++w) before += wc[w][k];
    if (bal[k] & (1u << lane))
      idx[off + before + __popc(bal[k] & ((1u << lane) - 1u))] = (int)(base + k * 256 + threadIdx.x);
  }
}

// Compacted operands Ac, Bc (ntot x p, column-major with an even leading
// dimension ld = ntot rounded up, the padding row zero, so that every column
// starts on a 16-byte boundary), residual norms, order.
__global__ void k_compact(const double* __restrict__ A, const double* __restrict__ B, long long n,
                          int p, const int* __restrict__ idx, const double* __restrict__ norm2,
                          QrState* st, double* __restrict__ Ac, double* __restrict__ Bc,
                          double* __restrict__ nu, double* __restrict__ nu0, int* __restrict__ pos,
                          int* __restrict__ perm, unsigned char* __restrict__ active) {
  const int ntot = st->ntot;
  const long long ld = ntot + (ntot & 1);
  if ((ntot & 1) && blockIdx.x == 0 && threadIdx.x == 0)
    for (int j = 0; j < p; ++j) Ac[ntot + j * ld] = Bc[ntot + j * ld] = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ntot; c += gridDim.x * blockDim.x) {
    const long long r = idx[c];
    for (int j = 0; j < p; ++j) {
      Ac[c + j * ld] = A[r + (long long)j * n];
      Bc[c + j * ld] = B[r + (long long)j * n];
    }
    const double v = sqrt(norm2[r]);
    nu[c] = v;
    nu0[c] = v;
    pos[c] = c;
    perm[c] = c;
    active[c] = 1;
  }
}

// The first step's candidates: one per block of 64 columns, none from recomputes.
__global__ void __launch_bounds__(64) k_first_best(const double* __restrict__ nu, int ntot,
                                                   int blocks, Best* __restrict__ best) {
  Best v{0.0, INT_MAX};
  const int c = blockIdx.x * 64 + threadIdx.x;
  if ((int)blockIdx.x < blocks && c < ntot) v = Best{nu[c], c};
  v = warp_best(v);
  __shared__ Best half;
  if (threadIdx.x == 32) half = v;
  __syncthreads();
  if (threadIdx.x == 0) best[blockIdx.x] = better(v, half);
}

// ------------------------------------------------------------- one pivot step
// The kernels of a step are resident while the one before them still writes
// (launch_early), so nothing that a step writes is read through a __restrict__
// pointer: read-only loads want data that no one changes in a kernel's lifetime.
// The pivot: the best of the blocks' candidates, its bookkeeping (one thread) and
// its feature vector x[i + j*p] = B(c, i) * A(c, j). The step number comes from the
// device, so that every step is the same launches and one graph serves them all; past
// the last step, or where no norm is left, it ends the loop.
__global__ void __launch_bounds__(1024) k_pick(int kmax, int p, int ld, int nbest,
                                               const Best* best, const double* __restrict__ Ac,
                                               const double* __restrict__ Bc, int* pos, int* perm,
                                               unsigned char* active, QrState* st, double* x,
                                               const LoopSignal sig) {
  after_previous();
  __shared__ int col;
  __shared__ Best warp_v[32];
  const int k = st->k;
  const bool run = !st->done && k < kmax;
  Best v{0.0, INT_MAX};
  if (run)
    for (int i = threadIdx.x; i < nbest; i += 1024) v = better(v, best[i]);
  v = warp_best(v);
  if ((threadIdx.x & 31) == 0) warp_v[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = warp_best(warp_v[threadIdx.x]);
    if (threadIdx.x == 0) {
      col = -1;
      if (run && v.nu > 0.0 && v.pos != INT_MAX) {
        const int q = v.pos;
        const int c = perm[q];
        const int ck = perm[k];
        perm[k] = c;
        perm[q] = ck;
        pos[ck] = q;
        pos[c] = k;
        active[c] = 0;
        col = c;
        st->k = k + 1;
        st->step = k;
      } else {
        if (run) st->done = 1;
        st->step = -1;
        loop_over(sig);
      }
      st->nrec = 0;
      loop_round(sig, ++st->rounds);
    }
  }
  __syncthreads();
  if (col < 0) return;
  const int m = p * p;
  for (int e = threadIdx.x; e < m; e += blockDim.x) {
    const int i = e % p, j = e / p;
    x[e] = Bc[col + (long long)i * ld] * Ac[col + (long long)j * ld];
  }
}

// cdot[l] = Q[:, l] . x for l < k: one block per l (a strided partial per
// thread, then a fixed-order tree), so the sums do not depend on scheduling.
__global__ void __launch_bounds__(256) k_qt_x(const double* Q, int m, const double* x,
                                              const QrState* st, double* cdot) {
  after_previous();
  const int l = blockIdx.x;
  if (l >= st->step) return;
  __shared__ double red[8];
  const double* q = Q + (long long)l * m;
  double s = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < m; i += 256) s = fma(q[i], x[i], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = red[0];
    for (int w = 1; w < 8; ++w) v += red[w];
    cdot[l] = v;
  }
}

// x -= Q[:, 0:k] cdot: a block takes kMinusRows consecutive rows, its 32 groups of
// as many lanes the columns l = w (mod 32), and the 32 partials are added in group
// order. Q streams from L2 (4.9 MB at 961 features and 640 pivots); eight rows a
// block spread it over 121 SMs (32 rows left 31 SMs to do it: 5.3 us a pass).
constexpr int kMinusRows = 8;
__global__ void __launch_bounds__(32 * kMinusRows) k_x_minus_qc(const double* Q, int m,
                                                                const double* cdot,
                                                                const QrState* st, double* x) {
  after_previous();
  const int k = st->step;
  if (k <= 0) return;
  __shared__ double red[32][kMinusRows + 1];
  const int r = threadIdx.x % kMinusRows, w = threadIdx.x / kMinusRows;
  const int i = blockIdx.x * kMinusRows + r;
  double s = 0.0;
  if (i < m) {
#pragma unroll 10
    for (int l = w; l < k; l += 32) s = fma(Q[i + (long long)l * m], cdot[l], s);
  }
  red[w][r] = s;
  __syncthreads();
  if (w == 0 && i < m) {
    double v = red[0][r];
#pragma unroll
    for (int u = 1; u < 32; ++u) v += red[u][r];
    x[i] -= v;
  }
}

// q_k = x / |x| into Q[:, k] and into Qm (depth-major: Qm[i*ldq + j] = q[i + j*p]).
__global__ void __launch_bounds__(1024) k_normalise(int p, int ldq, const double* x, QrState* st,
                                                    double* __restrict__ Q,
                                                    double* __restrict__ Qm) {
  after_previous();
  const int k = st->step;
  if (k < 0 || st->done) return;
  const int m = p * p;
  __shared__ double red[32];
  double s = 0.0;
  for (int e = threadIdx.x; e < m; e += blockDim.x) s = fma(x[e], x[e], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const double nrm = sqrt(red[0]);
  if (!(nrm > 0.0)) {
    if (threadIdx.x == 0) st->done = 1;
    return;
  }
  const double inv = 1.0 / nrm;
  for (int e = threadIdx.x; e < m; e += blockDim.x) {
    const double q = x[e] * inv;
    Q[(long long)k * m + e] = q;
    const int i = e % p, j = e / p;
    Qm[i * ldq + j] = q;
  }
}

// Residual-norm downdate of every active column with t_c = q_k . x_c, and the
// block's candidate for the next pivot, on the warp-specialised tile: 64 rows x
// BN columns, BN = p rounded up to a multiple of 8, four DMMA warps of 16 full rows
// each, so the row dot with A closes inside a quad of lanes. Qm's rows are
// ldq = p rounded up to even long (16-byte aligned for an odd p as well: on a 48^3
// grid with p = 31 the 128-column tile that odd p took until then ran 44 us a step,
// this one 17). An odd last row copies its zero padding partner.
template <int BN>
using UpdTile = dmma::WsTile<64, BN, 4, 1, 16, 3>;
// CTAs per SM while the accumulators (and, for the narrow tiles, the columns of A
// read ahead of the dot) leave registers: a narrow tile's CTA is short, and its
// loads' latency is what it waits for. 200 pivots on 48^3 points with four CTAs against
// three: 10.2 and 11.2 ms at p = 31, 13.4 and 14.4 at 38, 13.8 and 14.0 at 46; with three
// against two: 35.3 and 39.2 at 94, 48.3 and 48.6 at 110, 76.0 and 59.0 at 126.
template <int BN>
struct UpdMinBlocks {
  static constexpr int value = BN <= 40 ? 4 : BN <= 96 ? 3 : 2;
};
// Widest tile whose columns of A are read ahead: with and without 10.1 and 10.4 ms at
// p = 31, 13.4 and 13.7 at 38, 14.4 and 14.0 at 46, 22.8 and 21.6 at 62.
constexpr int kUpdAhead = 40;

template <int BN, int MINB>
__global__ void __launch_bounds__(UpdTile<BN>::THREADS, MINB)
    k_update_ws(const double* __restrict__ Ac, const double* __restrict__ Bc, int ntot, int ld,
                int p, int ldq,
                const double* Qm, const unsigned char* active, const int* pos, double* nu,
                double* nu0, QrState* st, int* rec_list, Best* best, int* err) {
  using T = UpdTile<BN>;
  extern __shared__ __align__(128) double smem[];
  const int m0 = blockIdx.x * T::BM;
  const int m_rem = min(T::BM, ntot - m0);
  T tile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  constexpr bool kAhead = BN <= kUpdAhead;
  double av[2][kAhead ? T::NT : 1][2];
  auto load_a = [&](int h, int j, int e) -> double {
    const int r = warp * 16 + g + 8 * h, c = j * 8 + 2 * t + e;
    return r < m_rem && c < p ? Ac[(m0 + r) + (long long)c * ld] : 0.0;
  };
  if (kAhead && !T::producer()) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < (kAhead ? T::NT : 1); ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) av[h][j][e] = load_a(h, j, e);
  }
  after_previous();  // (A does not change from step to step)
  if (st->step < 0 || st->done) return;
  const bool ok = tile.run(smem, Bc + m0, ld, (m_rem + 1) & ~1, Qm, ldq, p, p, err);
  if (T::producer()) return;
  Best v{0.0, INT_MAX};
  // a warp whose wait ran out has no product, but the others may have theirs and
  // wait for it at the barrier below
#pragma unroll
  for (int h = 0; ok && h < 2; ++h) {
    const int r = warp * 16 + g + 8 * h;
    double s = 0.0;
    if (r < m_rem) {
#pragma unroll
      for (int j = 0; j < T::NT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (j * 8 + 2 * t + e < p)
            s = fma(kAhead ? av[h][kAhead ? j : 0][e] : load_a(h, j, e), tile.acc[0][j][2 * h + e], s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (t == 0 && r < m_rem) {
      const int c = m0 + r;
      if (active[c] && downdate_norm(c, s, nu, nu0, st, rec_list))
        v = better(v, Best{nu[c], pos[c]});
    }
  }
  v = warp_best(v);
  __shared__ Best warp_v[T::NW];
  if (lane == 0) warp_v[warp] = v;
  asm volatile("bar.sync 1, %0;" ::"n"(T::NW * 32) : "memory");  // the DMMA warps
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < T::NW; ++w) v = better(v, warp_v[w]);
    best[blockIdx.x] = v;
  }
}

// Exact residual norms of the columns the downdate flagged in this step
// (dgeqpf's recompute). One CTA per flagged column at a time: the column's
// features x[i + j*p] = B(c, i) A(c, j) go to shared memory, are projected
// on q_0..q_k twice (classical Gram-Schmidt: all k+1 dots, one warp per q_l
// with a fixed lane order, then the update, one thread per feature summing
// over l in order), and the residual's norm becomes nu[c] and the new
// reference nu0[c]. cbuf: gridDim.x x kmax doubles of scratch for the dots. Every
// block leaves its candidate for the next pivot.
__global__ void __launch_bounds__(256) k_recompute(const double* __restrict__ Ac,
                                                   const double* __restrict__ Bc, int ld, int p,
                                                   const double* Q, int m, int kmax,
                                                   const int* rec_list, const int* pos, double* nu,
                                                   double* nu0, QrState* st, double* cbuf,
                                                   Best* best) {
  after_previous();
  extern __shared__ double x[];  // m features
  __shared__ double red[8];
  const int k1 = st->step + 1;
  if (k1 <= 0 || st->done) return;
  const int nrec = st->nrec;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* c = cbuf + (size_t)blockIdx.x * kmax;
  Best found{0.0, INT_MAX};  // thread 0: the block's candidate
  for (int f = blockIdx.x; f < nrec; f += gridDim.x) {
    const int col = rec_list[f];
    for (int e = threadIdx.x; e < m; e += 256) {
      const int i = e % p, j = e / p;
      x[e] = Bc[col + (long long)i * ld] * Ac[col + (long long)j * ld];
    }
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
      for (int l = warp; l < k1; l += 8) {
        const double* q = Q + (long long)l * m;
        double s = 0.0;
        for (int i = lane; i < m; i += 32) s = fma(q[i], x[i], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) c[l] = s;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < m; i += 256) {
        double s = 0.0;
        for (int l = 0; l < k1; ++l) s = fma(Q[(long long)l * m + i], c[l], s);
        x[i] -= s;
      }
      __syncthreads();
    }
    double s = 0.0;
    for (int i = threadIdx.x; i < m; i += 256) s = fma(x[i], x[i], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < 8; ++w) t += red[w];
      const double v = sqrt(t);
      nu[col] = v;
      nu0[col] = v;
      found = better(found, Best{v, pos[col]});
      atomicAdd(&st->total_rec, 1);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) best[blockIdx.x] = found;
}

// Householder QR of the K x p draws (host, FP64): returns p orthonormal columns
// spanning the same space, row-major (K x p) for the depth-major GEMM operand.
std::vector<double> orthonormal_rows(const std::vector<double>& g_colmajor, int K, int p) {
  std::vector<double> a = g_colmajor;  // column-major K x p
  std::vector<double> tau(p, 0.0);
  for (int j = 0; j < p; ++j) {
    double nrm = 0.0;
    for (int i = j; i < K; ++i) nrm += a[i + (size_t)j * K] * a[i + (size_t)j * K];
    nrm = std::sqrt(nrm);
    const double a0 = a[j + (size_t)j * K];
    const double beta = a0 >= 0 ? -nrm : nrm;
    if (nrm == 0.0) continue;
    const double v0 = a0 - beta;
    for (int i = j + 1; i < K; ++i) a[i + (size_t)j * K] /= v0;
    tau[j] = (beta - a0) / beta;
    a[j + (size_t)j * K] = beta;
    for (int c = j + 1; c < p; ++c) {
      double s = a[j + (size_t)c * K];
      for (int i = j + 1; i < K; ++i) s += a[i + (size_t)j * K] * a[i + (size_t)c * K];
      s *= tau[j];
      a[j + (size_t)c * K] -= s;
      for (int i = j + 1; i < K; ++i) a[i + (size_t)c * K] -= s * a[i + (size_t)j * K];
    }
  }
  // Q = H_0 ... H_{p-1} I[:, 0:p]
  std::vector<double> q((size_t)K * p, 0.0);
  for (int j = 0; j < p; ++j) q[j + (size_t)j * K] = 1.0;
  for (int j = p - 1; j >= 0; --j) {
    for (int c = 0; c < p; ++c) {
      double s = q[j + (size_t)c * K];
      for (int i = j + 1; i < K; ++i) s += a[i + (size_t)j * K] * q[i + (size_t)c * K];
      s *= tau[j];
      q[j + (size_t)c * K] -= s;
      for (int i = j + 1; i < K; ++i) q[i + (size_t)c * K] -= s * a[i + (size_t)j * K];
    }
  }
  std::vector<double> rows((size_t)K * p);
  for (int i = 0; i < K; ++i)
    for (int j = 0; j < p; ++j) rows[(size_t)i * p + j] = q[i + (size_t)j * K];
  return rows;
}

// srand48 Gaussian draws as include/common/utility.hpp:455-471: column-major.
std::vector<double> gaussian_draws(int m, int n) {
  std::vector<double> g((size_t)m * n);
  const double pi = 3.14159265358979323846;
  for (auto& v : g) {
    const double a = drand48(), b = drand48();
    v = std::sqrt(-2.0 * std::log(a)) * std::cos(2.0 * pi * b);
  }
  return g;
}

struct QrBuffers {
  double *A, *B, *norm2, *Ac, *Bc, *nu, *nu0, *Q, *Qm, *x, *cdot, *G1, *G2, *rec_dots;
  int *idx, *pos, *perm, *tile_cnt, *rec_list;
  Best* best;  // candidates: one per 64 columns, then one per recompute block
  unsigned char* active;
  QrState* st;
  int* err;  // a bounded pipeline wait of the update ran out
};

QrBuffers carve(Arena& a, long long n, int p, int k1, int k2, int kmax) {
  QrBuffers b;
  const int m = p * p;
  const int ntiles = (int)((n + 1023) / 1024);
  b.A = a.take<double>((size_t)n * p);
  b.B = a.take<double>((size_t)n * p);
  b.norm2 = a.take<double>((size_t)n);
  b.Ac = a.take<double>((size_t)(n + 1) * p);  // leading dimension up to n + 1 (even)
  b.Bc = a.take<double>((size_t)(n + 1) * p);
  b.nu = a.take<double>((size_t)n);
  b.nu0 = a.take<double>((size_t)n);
  b.Q = a.take<double>((size_t)m * kmax);
  b.Qm = a.take<double>((size_t)p * (p + (p & 1)));
  b.x = a.take<double>((size_t)m);
  b.cdot = a.take<double>((size_t)kmax);
  b.G1 = a.take<double>((size_t)k1 * p);
  b.G2 = a.take<double>((size_t)k2 * p);
  b.idx = a.take<int>((size_t)n);
  b.pos = a.take<int>((size_t)n);
  b.perm = a.take<int>((size_t)n);
  b.tile_cnt = a.take<int>((size_t)ntiles);
  b.rec_list = a.take<int>((size_t)n);
  b.rec_dots = a.take<double>((size_t)kRecomputeGrid * kmax);
  b.active = a.take<unsigned char>((size_t)n);
  b.best = a.take<Best>((size_t)((n + 63) / 64 + kRecomputeGrid));
  b.st = a.take<QrState>(1);
  b.err = a.take<int>(1);
  return b;
}

int set_update_attrs() {
  std::lock_guard<std::mutex> attr_lock(attr_mutex());
  static bool done[64] = {};
  int dev = 0;
  ISDF_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && done[dev]) return ISDF_OK;
  ISDF_CUDA(cudaFuncSetAttribute(k_recompute, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kMaxPre * kMaxPre)));
#define ISDF_UPD_ATTR(BN)                                                                  \
  ISDF_CUDA(cudaFuncSetAttribute(k_update_ws<BN, UpdMinBlocks<BN>::value>,                   \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,                \
                                 (int)UpdTile<BN>::SMEM_BYTES))
  ISDF_UPD_ATTR(16);
  ISDF_UPD_ATTR(24);
  ISDF_UPD_ATTR(32);
  ISDF_UPD_ATTR(40);
  ISDF_UPD_ATTR(48);
  ISDF_UPD_ATTR(56);
  ISDF_UPD_ATTR(64);
  ISDF_UPD_ATTR(72);
  ISDF_UPD_ATTR(80);
  ISDF_UPD_ATTR(88);
  ISDF_UPD_ATTR(96);
  ISDF_UPD_ATTR(104);
  ISDF_UPD_ATTR(112);
  ISDF_UPD_ATTR(120);
  ISDF_UPD_ATTR(128);
#undef ISDF_UPD_ATTR
  if (dev >= 0 && dev < 64) done[dev] = true;
  return ISDF_OK;
}

template <int BN>
void launch_update_bn(const QrBuffers& b, int ntot, int ld, int p, LoopQueue& q) {
  using T = UpdTile<BN>;
  const unsigned grid = (unsigned)((ntot + T::BM - 1) / T::BM);
  launch_early(k_update_ws<BN, UpdMinBlocks<BN>::value>, grid, T::THREADS, T::SMEM_BYTES, q, b.Ac,
               b.Bc, ntot, ld, p, p + (p & 1), b.Qm, b.active, b.pos, b.nu, b.nu0, b.st,
               b.rec_list, b.best, b.err);
}

// The downdate on the narrowest warp-specialised tile that holds p columns
// (p rounded up to a multiple of 8).
void launch_update_ws(const QrBuffers& b, int ntot, int ld, int p, LoopQueue& q) {
  switch ((p + 7) / 8) {
    case 0: case 1: case 2: launch_update_bn<16>(b, ntot, ld, p, q); break;
    case 3: launch_update_bn<24>(b, ntot, ld, p, q); break;
    case 4: launch_update_bn<32>(b, ntot, ld, p, q); break;
    case 5: launch_update_bn<40>(b, ntot, ld, p, q); break;
    case 6: launch_update_bn<48>(b, ntot, ld, p, q); break;
    case 7: launch_update_bn<56>(b, ntot, ld, p, q); break;
    case 8: launch_update_bn<64>(b, ntot, ld, p, q); break;
    case 9: launch_update_bn<72>(b, ntot, ld, p, q); break;
    case 10: launch_update_bn<80>(b, ntot, ld, p, q); break;
    case 11: launch_update_bn<88>(b, ntot, ld, p, q); break;
    case 12: launch_update_bn<96>(b, ntot, ld, p, q); break;
    case 13: launch_update_bn<104>(b, ntot, ld, p, q); break;
    case 14: launch_update_bn<112>(b, ntot, ld, p, q); break;
    case 15: launch_update_bn<120>(b, ntot, ld, p, q); break;
    default: launch_update_bn<128>(b, ntot, ld, p, q); break;
  }
}

}  // namespace

int qrcp_num_pre(int mu, double factor) { return iround(std::sqrt(mu * factor)); }

size_t qrcp_workspace_bytes(long long ng, int nstate, int mu, double factor) {
  const int p = qrcp_num_pre(mu, factor);
  Arena a;
  a.counting = true;
  carve(a, ng, p, nstate, nstate, std::min(mu, p * p));
  return a.off;
}

int qrcp_select(const QrcpArgs& args, Arena& arena, cudaStream_t s, QrcpResult* res) {
  const long long n = args.ng;
  const int p = qrcp_num_pre(args.mu, args.factor);
  const int k1 = args.nv1 + args.nc1, k2 = args.nv2 + args.nc2;
  if (p > args.nstate)
    return record_error(ISDF_ERR_ARG,
                        "numMu is too large for interpolative separable density fitting!");
  if ((long long)p * p > n)
    return record_error(ISDF_ERR_ARG, "numPre*numPre > ntot. The number of grid points is perhaps too small!");
  if (p > k1 || p > k2)
    return record_error(ISDF_ERR_UNSUPPORTED, "QRCP: numPre exceeds a state window");
  if (p > kMaxPre) return record_error(ISDF_ERR_UNSUPPORTED, "QRCP: numPre above 128");
  if (n > 0x7fffffffLL) return record_error(ISDF_ERR_UNSUPPORTED, "QRCP: Ng >= 2^31");
  const int m = p * p;
  const int kmax_cap = std::min(args.mu, m);
  QrBuffers b = carve(arena, n, p, k1, k2, kmax_cap);
  if (arena.overflowed()) return record_error(ISDF_ERR_NOMEM, "QRCP: workspace too small");
  ISDF_TRY(set_update_attrs());
  int launches = 0;

  // sketch (host): srand48(seed), G1 then G2, orthonormal columns
  srand48((long)args.seed);
  std::vector<double> g1 = gaussian_draws(k1, p);
  std::vector<double> g2 = gaussian_draws(k2, p);
  std::vector<double> q1 = orthonormal_rows(g1, k1, p);
  std::vector<double> q2 = orthonormal_rows(g2, k2, p);
  ISDF_CUDA(cudaMemcpyAsync(b.G1, q1.data(), sizeof(double) * q1.size(), cudaMemcpyHostToDevice, s));
  ISDF_CUDA(cudaMemcpyAsync(b.G2, q2.data(), sizeof(double) * q2.size(), cudaMemcpyHostToDevice, s));
  ISDF_CUDA(cudaMemsetAsync(b.st, 0, sizeof(QrState), s));
  ISDF_CUDA(cudaMemsetAsync(b.err, 0, sizeof(int), s));

  // A = psi_S1 G1, B = psi_S2 G2
  ISDF_TRY(dgemm_store((int)n, p, k1, args.d_psi + (long long)(args.nocc - args.nv1) * n, n, b.G1,
                       p, b.A, n, s));
  ISDF_TRY(dgemm_store((int)n, p, k2, args.d_psi + (long long)(args.nocc - args.nv2) * n, n, b.G2,
                       p, b.B, n, s));
  launches += 2;

  // norms, filter, compaction
  const int ntiles = (int)((n + 1023) / 1024);
  k_mg_norm<<<kNumSMs * 8, 256, 0, s>>>(b.A, b.B, n, p, b.norm2, b.st);
  k_keep_count<<<ntiles, 256, 0, s>>>(b.norm2, n, b.st, b.tile_cnt);
  k_scan_tiles<<<1, 1024, 0, s>>>(b.tile_cnt, ntiles, &b.st->ntot);
  k_keep_scatter<<<ntiles, 256, 0, s>>>(b.norm2, n, b.st, b.tile_cnt, b.idx);
  k_compact<<<kNumSMs * 4, 256, 0, s>>>(b.A, b.B, n, p, b.idx, b.norm2, b.st, b.Ac, b.Bc, b.nu,
                                        b.nu0, b.pos, b.perm, b.active);
  launches += 5;
  ISDF_CHECK_LAUNCH();
  QrState hst;
  ISDF_TRY(read_back(&hst, b.st, sizeof(QrState), s));
  const int ntot = hst.ntot;
  const int kmax = std::min(kmax_cap, ntot);
  res->ntot_mg = ntot;

  // pivoted Gram-Schmidt over the kept columns
  const int ld = ntot + (ntot & 1);  // Ac / Bc leading dimension (k_compact)
  const int ldq = p + (p & 1);
  const int ublocks = (ntot + 63) / 64, nbest = ublocks + kRecomputeGrid;
  // the first candidates: one per 64 columns, none from recomputes
  ISDF_CUDA(cudaMemsetAsync(b.best, 0, sizeof(Best) * (size_t)nbest, s));
  if (ublocks > 0) k_first_best<<<ublocks, 64, 0, s>>>(b.nu, ntot, ublocks, b.best);
  // One pivot step; the step number lives on the device.
  auto step = [&](LoopQueue& q, const LoopSignal& sig) {
    launch_early(k_pick, 1, 1024, 0, q, kmax, p, ld, nbest, b.best, b.Ac, b.Bc, b.pos, b.perm,
                 b.active, b.st, b.x, sig);
    for (int pass = 0; pass < 2; ++pass) {
      launch_early(k_qt_x, kmax, 256, 0, q, b.Q, m, b.x, b.st, b.cdot);
      launch_early(k_x_minus_qc, (m + kMinusRows - 1) / kMinusRows, 32 * kMinusRows, 0, q, b.Q, m,
                   b.cdot, b.st, b.x);
    }
    launch_early(k_normalise, 1, 1024, 0, q, p, ldq, b.x, b.st, b.Q, b.Qm);
    launch_update_ws(b, ntot, ld, p, q);
    launch_early(k_recompute, kRecomputeGrid, 256, sizeof(double) * m, q, b.Ac, b.Bc, ld, p, b.Q,
                 m, kmax_cap, b.rec_list, b.pos, b.nu, b.nu0, b.st, b.rec_dots, b.best + ublocks);
  };
  ISDF_CHECK_LAUNCH();
  Loop loop(s);
  if (kmax > 0) {
    // (launched one by one, the eight kernels of a step took the host longer than the
    // GPU at numPre = 31)
    constexpr int kBodySteps = 4, kSlackSteps = 2, kAheadSteps = 8;
    ISDF_TRY(loop.start(std::min(kmax, kAheadSteps), step));
    ISDF_TRY(loop.finish(kmax, kBodySteps, kSlackSteps, step, [&](bool* over) -> int {
      ISDF_TRY(read_back(&hst, b.st, sizeof(QrState), s));
      *over = hst.done != 0;
      return ISDF_OK;
    }));
    launches += 8 * kmax + 1;
  }
  ISDF_CHECK_LAUNCH();

  // piv = MGIdx[pivots], then the remaining kept columns in pivoted order, then 0
  std::vector<int> idx(ntot), perm(ntot);
  ISDF_TRY(read_back(&hst, b.st, sizeof(QrState), s));
  int err = 0;
  ISDF_TRY(read_back(&err, b.err, sizeof(int), s));
  if (err) return record_error(ISDF_ERR_TIMEOUT, "QRCP: an update pipeline wait timed out");
  if (hst.k != kmax && !hst.done) return record_error(ISDF_ERR_CUDA, "QRCP: steps are missing");
  ISDF_TRY(read_back(idx.data(), b.idx, sizeof(int) * ntot, s));
  ISDF_TRY(read_back(perm.data(), b.perm, sizeof(int) * ntot, s));
  std::memset(args.piv, 0, sizeof(int) * (size_t)n);
  for (int j = 0; j < ntot; ++j) args.piv[j] = idx[perm[j]];
  res->steps = kmax;
  res->num_pre = p;
  res->recomputes = hst.total_rec;
  res->done_early = hst.done;
  res->launches = launches + (readback_mailbox() ? (ntot > 0 ? 5 : 3) : 0);
  return ISDF_OK;
}

}  // namespace isdf_b200
