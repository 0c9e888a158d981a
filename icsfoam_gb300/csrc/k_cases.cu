// Independent cases stacked in one handle: the batch of many small cases as a
// leading dimension.
//
// The handle's mesh is the disjoint union of the cases' meshes (case k owns
// cells start[k] .. start[k+1]-1; no face joins two cases), so every
// cell- and face-parallel kernel of the pseudo iteration (fields, gradients,
// fluxes, cell residual, Jacobian rows, SpMV, LU-SGS levels, update) already
// treats each case exactly as a handle of its own would, and runs once for
// all of them.  What couples the cells of one system are the scalars of its
// GMRES (gmres.C:772-1107): the dot products and norms, the Hessenberg
// matrix, the Givens rotations, the back substitution, the stop test
// (coupledMatrixSolver.C:198-221) and the norm factors (gmres.C:812-850).
// Here each of those is per case:
//   * the Gram-Schmidt of a case of up to COLUMN_CELLS cells runs in a cluster
//     of blocks of its own (k_ccolumn); every other reduction runs over
//     segments of at most SEG_CELLS cells that never straddle two cases, and
//     the last segment of a case to finish folds the case's partial sums in
//     segment order.  Either way a case's sums depend only on its own cells
//     and sizes, not on the other cases in the stack;
//   * the Krylov scalars (H, c, s, bh, y, beta) live per case in device
//     memory and the per-case kernels read them there, so one restart cycle
//     is one launch sequence for all cases, captured once as a CUDA graph;
//   * the host reads every case's L1 residuals after a cycle and applies the
//     stop test per case; a case that has stopped (or broken down) is marked
//     inactive and its correction is left as it stands while the others go
//     on.
// The LU-SGS preconditioner, the SpMV and the fused operator passes are the
// handle's own (union) kernels: their rows only read rows of the same case.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "krylov.cuh"

namespace ics {

namespace {

constexpr int SEG_CELLS = 1024;  // cells per reduction segment (5120 vector entries)
constexpr int CB = 256;          // threads per segment block
// of the Gram-Schmidt steps, whose threads have all their loads in flight:
// 60 registers of entries at most
template <typename TV>
constexpr int MB = sizeof(TV) == 4 ? 256 : 512;
template <typename TV>
constexpr int MB_ENTRIES = 5 * SEG_CELLS / MB<TV>;
constexpr int PSTRIDE = 8;       // partial sums per segment
constexpr int HSTRIDE = MAX_DIRS * MAX_DIRS;

__device__ __forceinline__ bool case_on(const CaseDev& D, int c) { return D.active[c] && D.status[c] == 0; }

// Block-sum NV values, store them as this segment's partials, and on the
// last segment of case c to arrive fold the case's partials in segment order
// into out[0..NV).  True on thread 0 of that block.
template <int NV, int CB>
__device__ __forceinline__ bool case_finish(const CaseDev& D, int c, double (&v)[NV], double* __restrict__ out) {
  constexpr int G = FOLD_GROUP<NV>;
  __shared__ double sm[CB / 32][FOLD_VALUES<NV>];
  __shared__ bool amLast;
  const bool writer = threadIdx.x < 32 && threadIdx.x % G == 0 && threadIdx.x / G < NV;
  const int k = threadIdx.x / G;
  double s = block_sums<NV, CB / 32>(v, sm);
  const int s0 = D.caseSeg[c], ns = D.caseSeg[c + 1] - s0;
  if (ns > 1) {
    if (threadIdx.x < 32) {
      if (writer) {
        D.partials[(size_t)blockIdx.x * PSTRIDE + k] = s;
        __threadfence();
      }
      __syncwarp();
      if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(&D.counter[c], 1u);
        amLast = (t == (unsigned)ns - 1);
      }
    }
    __syncthreads();
    if (!amLast) return false;
    __threadfence();
    const volatile double* vp = D.partials;
    double acc[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) acc[q] = 0.0;
    for (int b = threadIdx.x; b < ns; b += CB)
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q] += vp[(size_t)(s0 + b) * PSTRIDE + q];
    s = block_sums<NV, CB / 32>(acc, sm);
    if (threadIdx.x == 0) D.counter[c] = 0;
  }
  if (threadIdx.x >= 32) return false;
  if (writer) out[k] = s;
  __syncwarp();
  return threadIdx.x == 0;
}

// start of a cycle for case c: beta = |w|, bh = (beta, 0, ...)
__device__ void case_beta0(const CaseDev& D, int c, double nrm2) {
  const double beta = sqrt(nrm2);
  D.beta[c] = beta;
  double* bh = D.bh + (size_t)c * (MAX_DIRS + 1);
  for (int i = 0; i <= D.m; ++i) bh[i] = 0.0;
  bh[0] = beta;
  if (!(beta > 0.0)) D.status[c] = isfinite(beta) ? 2 : 4;
}

// Hessenberg column i of case c, |w|^2 = nrm2
__device__ void case_hess(const CaseDev& D, int c, int i, double nrm2) {
  D.beta[c] = sqrt(nrm2);
  hess_column(D.H + (size_t)c * HSTRIDE, D.c + (size_t)c * MAX_DIRS, D.s + (size_t)c * MAX_DIRS,
              D.bh + (size_t)c * (MAX_DIRS + 1), i, D.m, nrm2);
}

// ------------------------------------------------- columns of small cases
// The Gram-Schmidt of a new Krylov vector against the basis and its
// normalisation (gmres.C:936-1011), one launch for all cases of up to
// COLUMN_CELLS cells:
//   for j = 0 .. dir:  h_j = w . v_j;  w -= h_j v_j
//   v_{dir+1} = w / |w|
// (dir = -1, the start of a cycle, has the last line only.)  A cluster of
// COLUMN_BLOCKS blocks holds a case's w in registers for the whole column and
// exchanges the blocks' sums of a step through distributed shared memory, so a
// step costs one cluster barrier and two FP64 folds instead of a launch with a
// reduction tail.  A case's sums depend only on its own size: the thread that
// takes an entry and the order of the sums are the same in every instance and
// every stack.  FP32 sums: a thread adds two runs of at most 16 products in
// FP32, everything across threads is FP64.  Further clusters rotate the cases'
// Hessenberg columns of the direction before, one block per case.
//
// The line is what the registers hold; below it the clusters were never the
// slower way (a solve of four cycles, us, clusters against steps of one launch,
// mixed / FP64: 2 cases of 1000 cells 324 : 441 / 407 : 633, 64 of 1000
// 720 : 730 / 1012 : 1048, 24 of 13000 1522 : 1949 / 2609 : 3202).  24 tubes
// of 480 to 12000 cells in mixed precision, a column of 5.5 steps on average:
// 13 us where the steps took 32, bound by the folds and the barrier (1500
// cycles a step) and, from 6000 cells on, the L2 reads of 8 SMs; in FP64 by the
// FP64 pipes of those 8 SMs.
constexpr int COLUMN_BLOCKS = 8;
constexpr int COLUMN_THREADS = 256;
constexpr int COLUMN_STRIDE = COLUMN_BLOCKS * COLUMN_THREADS;
constexpr int COLUMN_ROUNDS = 32;  // entries per thread at most
constexpr int COLUMN_CELLS = COLUMN_ROUNDS * COLUMN_STRIDE / 5;

__device__ __forceinline__ bool in_column(const CaseDev& D, int c) { return D.start[c + 1] - D.start[c] <= COLUMN_CELLS; }

template <typename TV, int K>
__global__ void __cluster_dims__(COLUMN_BLOCKS, 1, 1) __launch_bounds__(COLUMN_THREADS, sizeof(TV) * K <= 128 ? 2 : 1)
    k_ccolumn(CaseDev D, const TV* __restrict__ w, TV* __restrict__ V, long vs, int dir) {
  namespace cg = cooperative_groups;
  __shared__ TV sums[COLUMN_THREADS];
  __shared__ double slot[2][32];  // of the cluster's 8 x 4 folding warps
  __shared__ double result;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int c = blockIdx.x / COLUMN_BLOCKS;
  if (c >= D.n) {  // the rotations, not part of the exchange
    c = blockIdx.x - COLUMN_BLOCKS * D.n;
    if (tid == 0 && dir > 0 && c < D.n && in_column(D, c) && case_on(D, c)) case_hess(D, c, dir - 1, D.red[2 * c + ((dir - 1) & 1)]);
    return;
  }
  if (!in_column(D, c) || !case_on(D, c)) return;  // the whole cluster
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // the other blocks' shared memory exists after the wait
  const int rank = (int)cluster.block_rank();
  // this block's entries of the case start at first; a thread's follow at
  // COLUMN_STRIDE from its own, cnt of them
  const int first = rank * COLUMN_THREADS, n = 5 * (D.start[c + 1] - D.start[c]);
  const size_t e0 = 5 * (size_t)D.start[c] + first + tid;
  const int cnt = (n - first - tid + COLUMN_STRIDE - 1) / COLUMN_STRIDE;
  // rounds that hold any entry of the block: an FP64 instruction costs its
  // cycles with every lane predicated off too
  const int used = (n - first + COLUMN_STRIDE - 1) / COLUMN_STRIDE;
  TV x[K], v[K], vn[K];
  auto fetch = [&](TV (&r)[K], const TV* __restrict__ src) {
#pragma unroll
    for (int q = 0; q < K; ++q) r[q] = q < cnt ? src[q * COLUMN_STRIDE] : TV(0);
  };
  fetch(x, w + e0);
  if (dir >= 0) fetch(v, V + e0);
  cluster.barrier_wait();
  double total = 0.0;
#pragma unroll 1
  for (int j = 0; j <= dir + 1; ++j) {
    if (j < dir) fetch(vn, V + (size_t)(j + 1) * vs + e0);  // in flight during the exchange
    TV a0 = TV(0), a1 = TV(0);
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (q < used) {
        const TV y = j <= dir ? v[q] : x[q];
        if (q & 1)
          a1 = fma(x[q], y, a1);
        else
          a0 = fma(x[q], y, a0);
      }
    sums[tid] = a0 + a1;
    __syncthreads();
    if (warp < 4) {
      double s = widen(sums[tid]) + widen(sums[tid + 128]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane < COLUMN_BLOCKS) *cluster.map_shared_rank(&slot[j & 1][4 * rank + warp], lane) = s;
    }
    // the slots of step j are written again in step j + 2, after every block
    // has passed the barrier of step j + 1 and so has read them
    cluster.sync();
    if (warp == 0) {
      double s = slot[j & 1][lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) result = s;
    }
    __syncthreads();
    total = result;
    if (j <= dir) {
      const TV h = TV(total);
#pragma unroll
      for (int q = 0; q < K; ++q)
        if (q < used) {
          x[q] -= h * v[q];
          v[q] = vn[q];
        }
      if (rank == 0 && tid == 0) D.H[(size_t)c * HSTRIDE + j * D.m + dir] = total;
    }
  }
  if (rank == 0 && tid == 0) {
    D.red[2 * c + (dir & 1)] = total;  // the rotation of direction dir - 1 reads the other one meanwhile
    if (dir < 0) case_beta0(D, c, total);
  }
  // the next basis vector (the last direction of a cycle needs none)
  if (dir + 1 < D.m) {
    const TV b = TV(sqrt(total)), rb = TV(1) / b, rl = rb * fma(-b, rb, TV(1));
    TV* out = V + (size_t)(dir + 1) * vs + e0;
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (q < cnt) out[q * COLUMN_STRIDE] = quotient(x[q], rb, rl);
  }
}

// ------------------------------------------------- columns of large cases
// One pipelined modified Gram-Schmidt step per case of more than COLUMN_CELLS
// cells: w -= hprev vprev (when vprev), then the sum of w.vnext (or w.w) into
// H[outIdx] (outRed < 0) or red[outRed]; post 1 starts the cycle, post 2
// finishes Hessenberg column dir.
template <typename TV>
__global__ void __launch_bounds__(MB<TV>) k_cmgs(CaseDev D, TV* __restrict__ w, const TV* __restrict__ vprev,
                                             int hprevIdx, const TV* __restrict__ vnext, int outIdx, int outRed,
                                             int post, int dir) {
  const int c = D.segCase[blockIdx.x];
  if (in_column(D, c)) return;  // every segment of the case
  const bool on = case_on(D, c);
  double acc[1] = {0.0};
  if (on) {
    const size_t e0 = 5 * (size_t)D.segBeg[blockIdx.x] + threadIdx.x;
    const int n = 5 * (D.segEnd[blockIdx.x] - D.segBeg[blockIdx.x]) - threadIdx.x;  // entry q MB<TV> exists: q MB<TV> < n
    const TV h = vprev ? TV(D.H[(size_t)c * HSTRIDE + hprevIdx]) : TV(0);
    TV x[MB_ENTRIES<TV>], p[MB_ENTRIES<TV>], v[MB_ENTRIES<TV>];  // all loads of a thread in flight
#pragma unroll
    for (int q = 0; q < MB_ENTRIES<TV>; ++q) {
      const bool in = q * MB<TV> < n;
      x[q] = in ? w[e0 + q * MB<TV>] : TV(0);
      if (vprev) p[q] = in ? vprev[e0 + q * MB<TV>] : TV(0);
      if (vnext) v[q] = in ? vnext[e0 + q * MB<TV>] : TV(0);
    }
    TV t = TV(0);
#pragma unroll
    for (int q = 0; q < MB_ENTRIES<TV>; ++q) {
      if (vprev) {
        x[q] -= h * p[q];
        if (q * MB<TV> < n) w[e0 + q * MB<TV>] = x[q];
      }
      t += x[q] * (vnext ? v[q] : x[q]);
    }
    acc[0] = double(t);
  }
  double* out = outRed < 0 ? D.H + (size_t)c * HSTRIDE + outIdx : D.red + 2 * c + outRed;
  if (case_finish<1, MB<TV>>(D, c, acc, out) && on) {
    if (post == 1)
      case_beta0(D, c, *out);
    else if (post == 2)
      case_hess(D, c, dir, *out);
  }
}

// v = w / beta of the segment's case
template <typename TV>
__global__ void __launch_bounds__(MB<TV>) k_cscale(CaseDev D, const TV* __restrict__ w, TV* __restrict__ v) {
  const int c = D.segCase[blockIdx.x];
  if (in_column(D, c) || !case_on(D, c)) return;
  const TV b = TV(D.beta[c]), rb = TV(1) / b, rl = rb * fma(-b, rb, TV(1));
  const size_t e0 = 5 * (size_t)D.segBeg[blockIdx.x] + threadIdx.x;
  const int n = 5 * (D.segEnd[blockIdx.x] - D.segBeg[blockIdx.x]) - threadIdx.x;
  TV x[MB_ENTRIES<TV>];
#pragma unroll
  for (int q = 0; q < MB_ENTRIES<TV>; ++q) x[q] = q * MB<TV> < n ? w[e0 + q * MB<TV>] : TV(0);
#pragma unroll
  for (int q = 0; q < MB_ENTRIES<TV>; ++q)
    if (q * MB<TV> < n) v[e0 + q * MB<TV>] = quotient(x[q], rb, rl);
}

template <typename TV>
void column_small(Handle& h, cudaStream_t st, const TV* w, TV* V, long vs, int dir) {
  const CaseDev& D = h.cases.d;
  const int blocks = COLUMN_BLOCKS * (D.n + (D.n + COLUMN_BLOCKS - 1) / COLUMN_BLOCKS);
  const int rounds = (5 * h.cases.columnCells + COLUMN_STRIDE - 1) / COLUMN_STRIDE;
  auto launch = [&](auto kern) {
    ICS_LAUNCH(h, ICS_K_MGS, kern<<<blocks, COLUMN_THREADS, 0, st>>>(D, w, V, vs, dir));
  };
  if (rounds <= 4)
    launch(k_ccolumn<TV, 4>);
  else if (rounds <= 16)
    launch(k_ccolumn<TV, 16>);
  else
    launch(k_ccolumn<TV, COLUMN_ROUNDS>);
}

template <typename TV>
void column_large(Handle& h, TV* w, TV* V, long vs, int dir) {
  const CaseDev& D = h.cases.d;
  const int ns = h.cases.nseg, m = D.m;
  for (int j = 0; j <= dir; ++j)
    ICS_LAUNCH(h, ICS_K_MGS,
               k_cmgs<TV><<<ns, MB<TV>, 0, h.stream>>>(D, w, j > 0 ? V + (size_t)(j - 1) * vs : nullptr, (j - 1) * m + dir,
                                                   V + (size_t)j * vs, j * m + dir, -1, 0, dir));
  if (dir < 0)
    ICS_LAUNCH(h, ICS_K_MGS, k_cmgs<TV><<<ns, MB<TV>, 0, h.stream>>>(D, w, nullptr, 0, nullptr, 0, 0, 1, 0));
  else
    ICS_LAUNCH(h, ICS_K_MGS, k_cmgs<TV><<<ns, MB<TV>, 0, h.stream>>>(D, w, V + (size_t)dir * vs, dir * m + dir, nullptr, 0, 1,
                                                                 2, dir));
  if (dir + 1 < m)
    ICS_LAUNCH(h, ICS_K_VECTOR, k_cscale<TV><<<ns, MB<TV>, 0, h.stream>>>(D, w, V + (size_t)(dir + 1) * vs));
}

// the column of direction dir for every case, each by its own size; where a
// stack has both, the small ones' launch runs beside the large ones' steps
// (one after the other 31.5 ms for a step of 8 tubes of 1600 to 40000 cells,
// beside 29.0)
template <typename TV>
void case_column(Handle& h, TV* w, TV* V, long vs, int dir) {
  const CaseSet& S = h.cases;
  const bool beside = S.side && !h.prof;
  if (beside) {
    ICS_CUDA(cudaEventRecord(S.fork, h.stream));
    ICS_CUDA(cudaStreamWaitEvent(S.side, S.fork, 0));
  }
  if (S.columnCells) column_small<TV>(h, beside ? S.side : h.stream, w, V, vs, dir);
  if (S.columnLarge) column_large<TV>(h, w, V, vs, dir);
  if (beside) {
    ICS_CUDA(cudaEventRecord(S.join, S.side));
    ICS_CUDA(cudaStreamWaitEvent(h.stream, S.join, 0));
  }
}

// back substitution H y = bh per case (one warp per case)
__global__ void __launch_bounds__(128) k_cbacksub(CaseDev D) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= D.n || !case_on(D, c)) return;
  const int m = D.m;
  if (in_column(D, c)) {  // the last column is not rotated yet
    if ((threadIdx.x & 31) == 0) case_hess(D, c, m - 1, D.red[2 * c + ((m - 1) & 1)]);
    __syncwarp();
  }
  back_substitute(D.H + (size_t)c * HSTRIDE, D.bh + (size_t)c * (MAX_DIRS + 1), D.y + (size_t)c * MAX_DIRS, m);
}

// x += sum_i y_i V_i on the segment's case: XPARTS blocks per segment, so that a
// thread has five entries to wait for and not twenty (24 tubes of 480 to 12000
// cells, mixed: a time step with 24 of these launches 11.2 -> 10.7 ms)
constexpr int XPARTS = 4;
template <typename TV>
__global__ void __launch_bounds__(CB) k_cxupdate(CaseDev D, TV* __restrict__ x, const TV* __restrict__ V,
                                                 long vstride) {
  const int seg = blockIdx.x / XPARTS, part = blockIdx.x % XPARTS;
  const int c = D.segCase[seg];
  if (!case_on(D, c)) return;
  __shared__ TV y[MAX_DIRS];  // converted once, not per element
  if ((int)threadIdx.x < D.m) y[threadIdx.x] = convert<TV>(D.y[(size_t)c * MAX_DIRS + threadIdx.x]);
  __syncthreads();
  constexpr int SPAN = 5 * SEG_CELLS / XPARTS;
  const size_t e0 = 5 * (size_t)D.segBeg[seg] + part * SPAN + threadIdx.x;
  const int n = 5 * (D.segEnd[seg] - D.segBeg[seg]) - part * SPAN - threadIdx.x;  // entry q CB exists: q CB < n
  TV a[SPAN / CB];
#pragma unroll
  for (int q = 0; q < SPAN / CB; ++q) a[q] = q * CB < n ? x[e0 + q * CB] : TV(0);
#pragma unroll 2
  for (int i = 0; i < D.m; ++i) {
    const TV* v = V + (size_t)i * vstride + e0;
    const TV yi = y[i];
#pragma unroll
    for (int q = 0; q < SPAN / CB; ++q)
      if (q * CB < n) a[q] += yi * v[q * CB];
  }
#pragma unroll
  for (int q = 0; q < SPAN / CB; ++q)
    if (q * CB < n) x[e0 + q * CB] = a[q];
}

// r = b - t and the case's L1 sums per equation
template <typename TV>
__global__ void __launch_bounds__(CB) k_cresid(CaseDev D, const double* __restrict__ b, const TV* __restrict__ t,
                                               TV* __restrict__ r) {
  const int c = D.segCase[blockIdx.x];
  double acc[5] = {0, 0, 0, 0, 0};
  if (case_on(D, c)) {
    const int c1 = D.segEnd[blockIdx.x];
    for (int q = D.segBeg[blockIdx.x] + threadIdx.x; q < c1; q += CB)
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const TV v = convert<TV>(b[5 * q + k]) - t[5 * q + k];
        r[5 * q + k] = v;
        acc[k] += fabs(widen(v));
      }
  }
  case_finish<5, CB>(D, c, acc, D.res + 5 * c);
}

// per case: the norm-factor sums (rho, rhoE, |rhoU|) of |A (W - avg W)| + |b|
// and |b| per equation
template <typename TV>
__global__ void __launch_bounds__(CB) k_cnormfac(CaseDev D, const double* __restrict__ b, const TV* __restrict__ t) {
  const int c = D.segCase[blockIdx.x];
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int c1 = D.segEnd[blockIdx.x];
  for (int q = D.segBeg[blockIdx.x] + threadIdx.x; q < c1; q += CB) {
    const double t0 = widen(t[5 * q]), t4 = widen(t[5 * q + 4]);
    const double t1 = widen(t[5 * q + 1]), t2 = widen(t[5 * q + 2]), t3 = widen(t[5 * q + 3]);
    const double b0 = b[5 * q], b1 = b[5 * q + 1], b2 = b[5 * q + 2], b3 = b[5 * q + 3], b4 = b[5 * q + 4];
    acc[0] += fabs(t0) + fabs(b0);
    acc[1] += fabs(t4) + fabs(b4);
    acc[2] += sqrt(t1 * t1 + t2 * t2 + t3 * t3) + sqrt(b1 * b1 + b2 * b2 + b3 * b3);
    acc[3] += fabs(b0);
    acc[4] += fabs(b1);
    acc[5] += fabs(b2);
    acc[6] += fabs(b3);
    acc[7] += fabs(b4);
  }
  case_finish<8, CB>(D, c, acc, D.nfr + 8 * c);
}

// per case: the average of W per equation (gAverage)
__global__ void __launch_bounds__(CB) k_cwavg(CaseDev D, const double* __restrict__ W) {
  const int c = D.segCase[blockIdx.x];
  double acc[5] = {0, 0, 0, 0, 0};
  const int c1 = D.segEnd[blockIdx.x];
  for (int q = D.segBeg[blockIdx.x] + threadIdx.x; q < c1; q += CB)
#pragma unroll
    for (int k = 0; k < 5; ++k) acc[k] += W[5 * q + k];
  double* avg = D.avg + 5 * c;
  if (case_finish<5, CB>(D, c, acc, avg)) {
    const int nc = D.start[c + 1] - D.start[c];
    for (int k = 0; k < 5; ++k) avg[k] = avg[k] / nc;
  }
}

template <typename TV>
__global__ void __launch_bounds__(CB) k_cwmavg(CaseDev D, const double* __restrict__ W, TV* __restrict__ out) {
  const int c = D.segCase[blockIdx.x];
  const double* avg = D.avg + 5 * c;
  const int c1 = D.segEnd[blockIdx.x];
  for (int q = D.segBeg[blockIdx.x] + threadIdx.x; q < c1; q += CB)
#pragma unroll
    for (int k = 0; k < 5; ++k) out[5 * q + k] = convert<TV>(W[5 * q + k] - avg[k]);
}

// per case: sum of the cells' (R_rho V)^2
__global__ void __launch_bounds__(CB) k_cl2(CaseDev D, const double* __restrict__ a) {
  const int c = D.segCase[blockIdx.x];
  double acc[1] = {0.0};
  const int c1 = D.segEnd[blockIdx.x];
  for (int q = D.segBeg[blockIdx.x] + threadIdx.x; q < c1; q += CB) acc[0] += a[q];
  case_finish<1, CB>(D, c, acc, D.l2 + c);
}

template <typename TV>
__global__ void k_cto_dW(int N, const TV* __restrict__ x, double* __restrict__ dW, int s0, int s1, int s2) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  dW[5 * c] = widen(x[5 * c]);
  dW[5 * c + 1] = s0 == -1 ? 0.0 : widen(x[5 * c + 1]);
  dW[5 * c + 2] = s1 == -1 ? 0.0 : widen(x[5 * c + 2]);
  dW[5 * c + 3] = s2 == -1 ? 0.0 : widen(x[5 * c + 3]);
  dW[5 * c + 4] = widen(x[5 * c + 4]);
}

// coupledMatrix::solver::stop (coupledMatrixSolver.C:198-221) for one case
bool case_stop(const Handle& h, int nIter, const double* in, const double* fi) {
  const ics_config& c = h.cfg.c;
  if (nIter < c.min_iter) return false;
  double mx = -VGREAT, mrel = -VGREAT;
  for (int k = 0; k < 5; ++k) mx = fmax(mx, fi[k]);
  mrel = fmax(mrel, fi[0] / (in[0] + ROOTVSMALL));
  mrel = fmax(mrel, fi[4] / (in[4] + ROOTVSMALL));
  for (int k = 0; k < 3; ++k)
    if (h.m.solD[k] == 1) mrel = fmax(mrel, fi[1 + k] / (in[1 + k] + ROOTVSMALL));
  return nIter >= c.max_iter || mx < c.tolerance || mrel < c.rel_tol;
}

template <typename TV>
int gmres_cases_t(Handle& h, std::vector<int>& caseStatus) {
  CaseSet& S = h.cases;
  const int N = h.m.N, m = h.cfg.c.n_directions, n = S.n, ns = S.nseg;
  const long n5 = 5L * N;
  const long vs = (long)kstride(h);
  cudaStream_t st = h.stream;
  TV* V = (TV*)h.kv;
  TV* w = (TV*)h.kw;
  TV* x = (TV*)h.kx;
  TV* t = (TV*)h.kt;
  S.d.m = m;
  const CaseDev D = S.d;
  for (int k = 0; k < n; ++k) S.hactive[k] = S.frozen[k] ? 0 : 1;
  ICS_CUDA(cudaMemcpyAsync((void*)D.active, S.hactive, n * sizeof(int), cudaMemcpyHostToDevice, st));
  ICS_CUDA(cudaMemsetAsync(D.status, 0, n * sizeof(int), st));
  ICS_CUDA(cudaMemsetAsync(&h.ks->status, 0, sizeof(int), st));  // bounded waits of the sync-free sweeps
  // norm factors and initial residuals per case (gmres.C:812-850)
  ICS_LAUNCH(h, ICS_K_VECTOR, k_cwavg<<<ns, CB, 0, st>>>(D, h.W));
  ICS_LAUNCH(h, ICS_K_VECTOR, k_cwmavg<TV><<<ns, CB, 0, st>>>(D, h.W, w));
  spmv(h, w, t);
  ICS_LAUNCH(h, ICS_K_VECTOR, k_cnormfac<TV><<<ns, CB, 0, st>>>(D, h.src, t));
  ICS_CUDA(cudaMemcpyAsync(S.hnfr, D.nfr, 8ull * n * sizeof(double), cudaMemcpyDeviceToHost, st));
  ICS_CUDA(cudaStreamSynchronize(st));
  std::vector<double> nf(3 * n), fin(S.initRes);
  for (int k = 0; k < n; ++k) {
    const double* q = S.hnfr + 8 * k;
    for (int j = 0; j < 3; ++j) nf[3 * k + j] = q[j] + VSMALL;
    double* in = &S.initRes[5 * k];
    if (!S.hactive[k]) continue;
    in[0] = q[3] / nf[3 * k];
    in[1] = q[4] / nf[3 * k + 2];
    in[2] = q[5] / nf[3 * k + 2];
    in[3] = q[6] / nf[3 * k + 2];
    in[4] = q[7] / nf[3 * k + 1];
    std::copy(in, in + 5, &fin[5 * k]);
  }
  std::vector<int> nIter(n, 0);
  caseStatus.assign(n, ICS_OK);
  ICS_CUDA(cudaMemsetAsync(x, 0, n5 * sizeof(TV), st));
  to_vec(h, h.src, w);
  auto cycle = [&]() {
    precondition(h, w);
    case_column<TV>(h, w, V, vs, -1);
    for (int i = 0; i < m; ++i) {
      const TV* vi = V + (size_t)i * vs;
      if (!fused_operator(h, vi, w)) {
        spmv(h, vi, w);
        precondition(h, w);
      }
      case_column<TV>(h, w, V, vs, i);
    }
    ICS_LAUNCH(h, ICS_K_SCALAR, k_cbacksub<<<(n + 3) / 4, 128, 0, st>>>(D));
    ICS_LAUNCH(h, ICS_K_VECTOR, k_cxupdate<TV><<<XPARTS * ns, CB, 0, st>>>(D, x, V, vs));
    spmv(h, x, t);
    ICS_LAUNCH(h, ICS_K_VECTOR, k_cresid<TV><<<ns, CB, 0, st>>>(D, h.src, t, w));
  };
  // the captured launches hold DevMesh and CaseDev by value
  const int key = 30000000 + (h.m.vjslot ? 10000000 : 0) + h.cfg.c.preconditioner * 100000 + prec(h) * 1000 + m;
  const bool useGraph = !h.prof;
  if (useGraph && h.cycleKey != key) {
    drop_graphs(h);
    cudaGraph_t g = nullptr;
    const long long before = h.launches;
    ICS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    cycle();
    ICS_CUDA(cudaStreamEndCapture(st, &g));
    ICS_CUDA(cudaGraphInstantiate(&h.cycleExec, g, 0));
    ICS_CUDA(cudaGraphDestroy(g));
    h.cycleLaunches = h.launches - before;
    h.launches = before;
    h.cycleKey = key;
  }
  int status = ICS_OK;
  for (bool any = true; any;) {
    if (useGraph) {
      ICS_CUDA(cudaGraphLaunch(h.cycleExec, st));
      h.launches += h.cycleLaunches;
    } else {
      cycle();
    }
    ICS_CUDA(cudaGetLastError());
    int sweepStatus = 0;
    ICS_CUDA(cudaMemcpyAsync(S.hres, D.res, 5ull * n * sizeof(double), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaMemcpyAsync(S.hstatus, D.status, n * sizeof(int), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaMemcpyAsync(&sweepStatus, &h.ks->status, sizeof(int), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaStreamSynchronize(st));
    if (sweepStatus & 8) {
      status = ICS_ERR_TIMEOUT;
      break;
    }
    any = false;
    for (int k = 0; k < n; ++k) {
      if (!S.hactive[k]) continue;
      nIter[k]++;
      if (S.hstatus[k]) {
        caseStatus[k] = (S.hstatus[k] & 4) ? ICS_ERR_NONFINITE : ICS_ERR_BREAKDOWN;
        S.hactive[k] = 0;
        continue;
      }
      const double* rs = S.hres + 5 * k;
      double* fi = &fin[5 * k];
      bool finite = true;
      fi[0] = rs[0] / nf[3 * k];
      fi[4] = rs[4] / nf[3 * k + 1];
      for (int j = 0; j < 3; ++j) fi[1 + j] = h.m.solD[j] == -1 ? 0.0 : rs[1 + j] / nf[3 * k + 2];
      for (int j = 0; j < 5; ++j) finite = finite && std::isfinite(fi[j]);
      if (!finite) {
        caseStatus[k] = ICS_ERR_NONFINITE;
        S.hactive[k] = 0;
        continue;
      }
      if (case_stop(h, nIter[k], &S.initRes[5 * k], fi))
        S.hactive[k] = 0;
      else
        any = true;
    }
    if (any)
      ICS_CUDA(cudaMemcpyAsync((void*)D.active, S.hactive, n * sizeof(int), cudaMemcpyHostToDevice, st));
  }
  ICS_LAUNCH(h, ICS_K_VECTOR, k_cto_dW<TV><<<grid_for(N, 256), 256, 0, st>>>(N, x, h.dW, h.m.solD[0], h.m.solD[1],
                                                                             h.m.solD[2]));
  ICS_CUDA(cudaStreamSynchronize(st));
  for (int k = 0; k < n; ++k) {
    S.cycles[k] = S.frozen[k] ? 0 : nIter[k];
    if (!S.frozen[k]) std::copy(&fin[5 * k], &fin[5 * k] + 5, &S.finRes[5 * k]);
  }
  return status;
}

// the next 256-byte aligned array of count T at offset off of base
template <typename T>
T* carve(char* base, size_t& off, size_t count) {
  T* r = base ? reinterpret_cast<T*>(base + off) : nullptr;
  off += ((count * sizeof(T) + 255) / 256) * 256;
  return r;
}

}  // namespace

void free_cases(Handle& h) {
  CaseSet& S = h.cases;
  if (S.mem) cudaFree(S.mem);
  if (S.hres) cudaFreeHost(S.hres);
  if (S.fork) cudaEventDestroy(S.fork);
  if (S.join) cudaEventDestroy(S.join);
  if (S.side) cudaStreamDestroy(S.side);
  S = CaseSet();
  h.m.caseOf = nullptr;
  h.m.caseSer = nullptr;
}

void set_cases(Handle& h, int n, const int* start) {
  const int N = h.m.N;
  if (n < 1 || !start || start[0] != 0 || start[n] != N) throw std::string("case_start must run from 0 to n_cells");
  for (int k = 0; k < n; ++k)
    if (start[k + 1] <= start[k]) throw std::string("case_start must be strictly increasing");
  if (h.m.nInst > 1) throw std::string("stacked cases are not combined with Harmonic Balance");
  if (h.m.ncyc > 0) throw std::string("stacked cases carry no cyclic patches");
  if (h.cfg.c.solver != ICS_SOLVER_GMRES) throw std::string("stacked cases need the GMRES solver");
  if (h.scalarOn) throw std::string("stacked cases carry no passive scalar");
  std::vector<int> caseOf(N);
  for (int k = 0; k < n; ++k)
    for (int c = start[k]; c < start[k + 1]; ++c) caseOf[c] = k;
  if (h.m.F) {
    std::vector<int> own(h.m.F), nei(h.m.F);
    ICS_CUDA(cudaMemcpy(own.data(), h.m.own, h.m.F * sizeof(int), cudaMemcpyDeviceToHost));
    ICS_CUDA(cudaMemcpy(nei.data(), h.m.nei, h.m.F * sizeof(int), cudaMemcpyDeviceToHost));
    for (int f = 0; f < h.m.F; ++f)
      if (caseOf[own[f]] != caseOf[nei[f]]) throw std::string("an internal face joins two cases");
  }
  std::vector<int> segCase, segBeg, segEnd, caseSeg(n + 1);
  for (int k = 0; k < n; ++k) {
    caseSeg[k] = (int)segCase.size();
    for (int b = start[k]; b < start[k + 1]; b += SEG_CELLS) {
      segCase.push_back(k);
      segBeg.push_back(b);
      segEnd.push_back(std::min(b + SEG_CELLS, start[k + 1]));
    }
  }
  const int ns = (int)segCase.size();
  caseSeg[n] = ns;
  free_cases(h);
  drop_graphs(h);
  CaseSet& S = h.cases;
  CaseDev& D = S.d;
  D.n = n;
  D.m = h.cfg.c.n_directions;
  int *dSegCase, *dSegBeg, *dSegEnd, *dCaseSeg, *dStart;
  // one allocation, laid out twice: for its size, then over the allocation
  auto layout = [&](char* base) {
    size_t off = 0;
    dSegCase = carve<int>(base, off, ns);
    dSegBeg = carve<int>(base, off, ns);
    dSegEnd = carve<int>(base, off, ns);
    dCaseSeg = carve<int>(base, off, n + 1);
    dStart = carve<int>(base, off, n + 1);
    D.active = carve<int>(base, off, n);
    D.status = carve<int>(base, off, n);
    S.caseOf = carve<int>(base, off, N);
    D.counter = carve<unsigned int>(base, off, n);
    D.partials = carve<double>(base, off, (size_t)PSTRIDE * ns);
    D.H = carve<double>(base, off, (size_t)n * HSTRIDE);
    D.c = carve<double>(base, off, (size_t)n * MAX_DIRS);
    D.s = carve<double>(base, off, (size_t)n * MAX_DIRS);
    D.y = carve<double>(base, off, (size_t)n * MAX_DIRS);
    D.bh = carve<double>(base, off, (size_t)n * (MAX_DIRS + 1));
    D.beta = carve<double>(base, off, n);
    D.red = carve<double>(base, off, 2ull * n);
    D.res = carve<double>(base, off, 5ull * n);
    D.nfr = carve<double>(base, off, 8ull * n);
    D.avg = carve<double>(base, off, 5ull * n);
    D.l2 = carve<double>(base, off, n);
    S.ser = carve<double>(base, off, n);
    return off;
  };
  const size_t bytes = layout(nullptr);
  ICS_CUDA(cudaMalloc(&S.mem, bytes));
  ICS_CUDA(cudaMemsetAsync(S.mem, 0, bytes, h.stream));
  layout((char*)S.mem);
  ICS_CUDA(cudaMemcpyAsync(dSegCase, segCase.data(), ns * sizeof(int), cudaMemcpyHostToDevice, h.stream));
  ICS_CUDA(cudaMemcpyAsync(dSegBeg, segBeg.data(), ns * sizeof(int), cudaMemcpyHostToDevice, h.stream));
  ICS_CUDA(cudaMemcpyAsync(dSegEnd, segEnd.data(), ns * sizeof(int), cudaMemcpyHostToDevice, h.stream));
  ICS_CUDA(cudaMemcpyAsync(dCaseSeg, caseSeg.data(), (n + 1) * sizeof(int), cudaMemcpyHostToDevice, h.stream));
  ICS_CUDA(cudaMemcpyAsync(dStart, start, (n + 1) * sizeof(int), cudaMemcpyHostToDevice, h.stream));
  ICS_CUDA(cudaMemcpyAsync(S.caseOf, caseOf.data(), N * sizeof(int), cudaMemcpyHostToDevice, h.stream));
  ICS_CUDA(cudaStreamSynchronize(h.stream));
  D.segCase = dSegCase;
  D.segBeg = dSegBeg;
  D.segEnd = dSegEnd;
  D.caseSeg = dCaseSeg;
  D.start = dStart;
  // pinned mirrors: res [5n], nfr [8n], l2 [n], ser [n], status [n], active [n]
  ICS_CUDA(cudaMallocHost(&S.hres, sizeof(double) * 15ull * n + sizeof(int) * 2ull * n));
  S.hnfr = S.hres + 5 * n;
  S.hl2 = S.hnfr + 8 * n;
  S.hser = S.hl2 + n;
  S.hstatus = reinterpret_cast<int*>(S.hser + n);
  S.hactive = S.hstatus + n;
  S.n = n;
  S.nseg = ns;
  for (int k = 0; k < n; ++k) {
    const int cells = start[k + 1] - start[k];
    if (cells <= COLUMN_CELLS)
      S.columnCells = std::max(S.columnCells, cells);
    else
      S.columnLarge = true;
  }
  if (S.columnCells && S.columnLarge) {
    ICS_CUDA(cudaStreamCreateWithFlags(&S.side, cudaStreamNonBlocking));
    ICS_CUDA(cudaEventCreateWithFlags(&S.fork, cudaEventDisableTiming));
    ICS_CUDA(cudaEventCreateWithFlags(&S.join, cudaEventDisableTiming));
  }
  S.start.assign(start, start + n + 1);
  S.ctl.assign(n, PseudoControl());
  S.initRes.assign(5 * n, 0.0);
  S.prevRes.assign(5 * n, 0.0);
  S.finRes.assign(5 * n, 0.0);
  S.initValid.assign(n, 0);
  S.prevValid.assign(n, 0);
  S.frozen.assign(n, 0);
  S.cycles.assign(n, 0);
  h.m.caseOf = S.caseOf;
  h.m.caseSer = S.ser;
}

int gmres_cases(Handle& h, std::vector<int>& caseStatus) {
  return prec(h) == ICS_PREC_MIXED ? gmres_cases_t<float>(h, caseStatus) : gmres_cases_t<double>(h, caseStatus);
}

// per-case sums of (R_rho V)^2 from the last residual into the host mirror
void case_l2(Handle& h) {
  CaseSet& S = h.cases;
  ICS_LAUNCH(h, ICS_K_VECTOR, k_cl2<<<S.nseg, CB, 0, h.stream>>>(S.d, h.scratch));
  ICS_CUDA(cudaMemcpyAsync(S.hl2, S.d.l2, S.n * sizeof(double), cudaMemcpyDeviceToHost, h.stream));
  ICS_CUDA(cudaStreamSynchronize(h.stream));
}

// the cases' SER factors of the next residual (host mirror -> device)
void case_upload_ser(Handle& h) {
  CaseSet& S = h.cases;
  ICS_CUDA(cudaMemcpyAsync(S.ser, S.hser, S.n * sizeof(double), cudaMemcpyHostToDevice, h.stream));
}

}  // namespace ics
