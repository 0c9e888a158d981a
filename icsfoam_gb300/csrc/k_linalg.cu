// Block linear algebra on the sliced-ELL Jacobian and the Krylov solver.
//
//   spmv      y = A x, thread per row; diagonal + one 5x5 block per face slot,
//             slots in column order (= face order, the order Amul adds them)
//   lusgs     (D_s + L) D_s^-1 (D_s + U) z = r with the scalar diagonal D_s,
//             level-scheduled: a level holds rows whose lower (forward) or
//             upper (reverse) neighbours all lie in earlier levels.  Within a
//             row the neighbour contributions are subtracted in the order the
//             sequential sweep of lusgs.C:233-384 applies them.
//   jacobi    z = D^-1 r with precomputed 5x5 inverses (Jacobi.C:55-135)
//   gmres     left-preconditioned restarted GMRES with modified Gram-Schmidt
//             and Givens rotations (gmres.C:772-1107).  All vectors and the
//             Hessenberg matrix stay on the device.  The Gram-Schmidt sums are
//             exchanged through slots and added in slot order (k_column.cu),
//             the norms and residuals by a grid of the size's choosing whose
//             last block folds the partial sums in block order, so results are
//             reproducible run to run.  One host synchronisation per restart
//             cycle reads the L1 residuals for the stop test
//             (coupledMatrixSolver.C:198-221).
#include <algorithm>
#include <cmath>

#include "blocks.cuh"
#include "hb.cuh"
#include "ics_internal.cuh"
#include "krylov.cuh"

namespace ics {

// ------------------------------------------------------------------ reduce
constexpr int RB = 256;  // threads per reduction block

// Returns true on the one thread (thread 0 of the last block) that may read
// out[] then.
template <int NV>
__device__ __forceinline__ bool reduce_finish(double (&v)[NV], double* __restrict__ partials,
                                              unsigned int* __restrict__ counter, double* __restrict__ out) {
  constexpr int G = FOLD_GROUP<NV>;
  __shared__ double sm[RB / 32][FOLD_VALUES<NV>];
  __shared__ bool amLast;
  const int k = threadIdx.x / G;
  const bool writer = threadIdx.x < 32 && threadIdx.x % G == 0 && k < NV;
  double s = block_sums<NV, RB / 32>(v, sm);
  if (gridDim.x > 1) {
    if (threadIdx.x < 32) {
      if (writer) {
        partials[blockIdx.x * NV + k] = s;
        __threadfence();
      }
      __syncwarp();
      if (threadIdx.x == 0) amLast = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!amLast) return false;  // block-uniform: the last block folds all partials in a fixed order
    __threadfence();
    const volatile double* vp = partials;
    double acc[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) acc[q] = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += RB)
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q] += vp[b * NV + q];
    s = block_sums<NV, RB / 32>(acc, sm);
    if (threadIdx.x == 0) *counter = 0;
  }
  if (threadIdx.x >= 32) return false;
  if (writer) out[k] = s;
  __syncwarp();
  return threadIdx.x == 0;
}

// blocks of a reduction over n items: no more than hold one item per thread.
// A block's folds cost the same whatever it has summed, so idle blocks are not
// free: with 1216 blocks and a fold per value the residual of 10k cells took
// 31 us, and the 80 reductions and vector passes of a time step on 1000 cells
// 1.61 ms instead of 0.67
inline int reduce_grid(long n) { return (int)std::max(1L, std::min((long)REDUCE_BLOCKS, (n + RB - 1) / RB)); }
// blocks of an elementwise pass over n items
inline int pass_grid(long n) { return (int)std::max(1L, std::min(2L * REDUCE_BLOCKS, (n + RB - 1) / RB)); }

// ------------------------------------------------------------------- spmv
template <typename TB, typename TV>
__global__ void __launch_bounds__(128) k_spmv(DevMesh m, const TB* __restrict__ blk, const TB* __restrict__ dg,
                                              const TV* __restrict__ x, TV* __restrict__ y) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.N) return;
  const int s = c >> 5, lane = c & 31;
  TV xc[5], acc[5], part[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 5; ++k) xc[k] = x[5 * c + k];
  const TB* D = dg + (size_t)s * 25 * 32 + lane;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    TV a = TV(0);
#pragma unroll
    for (int j = 0; j < 5; ++j) a += TV(D[(5 * i + j) * 32]) * xc[j];
    acc[i] = a;
  }
  const int base = m.slot_base[s];
  const int ns = m.nslot[c];
  const TV g = TV(m.gamma);
#pragma unroll 1
  for (int t = 0; t < ns; ++t) {
    const int col = m.scol[(base + t) * 32 + lane];
    TV xj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xj[k] = x[5 * col + k];
    SlotBlock<TB> Bk;
    Bk.load(blk, base + t, lane);
    add_slot<1>(Bk, g, xj, acc, part, (t & 1) || t == ns - 1);
    if (m.vjslot) vj_sub<TB>(m, base + t, lane, col, xj, acc);
  }
  if (m.nInst > 1 && hb_in_zone(m, c)) {
    // Harmonic Balance coupling blocks V D_JK I with the other instances
    const int J = c / m.Nc, cl = c - J * m.Nc;
    const double Vc = m.V[c];
    for (int K = 0; K < m.nInst; ++K) {
      if (K == J) continue;
      const TV d = TV(Vc * m.Dhb[J * m.nInst + K]);
      const TV* xk = x + 5 * ((size_t)K * m.Nc + cl);
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] += d * xk[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) y[5 * c + k] = acc[k];
}

// Cyclic couplings (the interface part of Amul, blockFvMatrix.C:386-407):
// y_c += sum over the cyclic faces of c of B_f x_partner, B_f holding the
// partner's rotation; one thread per row that owns cyclic faces, after k_spmv.
template <typename TB, typename TV>
__global__ void __launch_bounds__(128) k_cyc_mv(DevMesh m, const TB* __restrict__ cblk, const TV* __restrict__ x,
                                                TV* __restrict__ y) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= m.ncrow) return;
  const int c = m.cyc_row[r];
  TV acc[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) acc[k] = y[5 * c + k];
  for (int e = m.cyc_ptr[r]; e < m.cyc_ptr[r + 1]; ++e) {
    const int pc = m.bpartner[m.cyc_face[e]];
    const TB* Bk = cblk + (size_t)e * 25;
    TV xj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xj[k] = x[5 * pc + k];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      TV a = TV(0);
#pragma unroll
      for (int j = 0; j < 5; ++j) a += TV(Bk[5 * i + j]) * xj[j];
      acc[i] += a;
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) y[5 * c + k] = acc[k];
}

// ------------------------------------- fused A x + LU-SGS (two-level schedule)
// On a schedule of two levels where the first holds the rows without lower
// neighbours and the second the rows without upper neighbours (the
// colour-blocked numbering of a bipartite mesh), z = M^-1 A x takes three
// passes instead of SpMV + two sweeps, and the second-level rows read their
// (lower) blocks once for both the product and the forward sweep:
//   pass 1 (level-0 rows): w = (A x)_c
//   pass 2 (level-1 rows): r' = (A x)_c - sum_lower L (rD w)_j, summed as
//                          D x_c + sum_lower L (x - rD w)_j;
//                          w_c = rD_c r'   (forward + fused first reverse)
//   pass 3 (level-0 rows): the reverse sweep, as k_lusgs_level MODE 1.
// Same arithmetic as the separate kernels up to the order of the sums.  In
// FP64 these passes are bound by the FP64 pipe, so their cost is their count
// of operations: one product per slot in pass 2 (98k rows: 94 -> 49 us) and
// products accumulated by multiply-adds over two slots (add_slot; pass 1 52 ->
// 40, pass 3 45 -> 43 us); the FP32 passes are bound by HBM and did not change.
template <typename TB, typename TV, int MINB = 1, int UNR = 1>
__global__ void __launch_bounds__(128, MINB) k_op_level0(DevMesh m, const TB* __restrict__ blk, const TB* __restrict__ dg,
                                                   const TV* __restrict__ x, TV* __restrict__ w,
                                                   const int* __restrict__ cells, int start, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int c = cells ? cells[start + i] : start + i;
  const int s = c >> 5, lane = c & 31;
  TV xc[5], acc[5], part[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 5; ++k) xc[k] = x[5 * (size_t)c + k];
  const TB* D = dg + (size_t)s * 25 * 32 + lane;
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    TV a = TV(0);
#pragma unroll
    for (int j = 0; j < 5; ++j) a += TV(D[(5 * r + j) * 32]) * xc[j];
    acc[r] = a;
  }
  const int base = m.slot_base[s];
  const int ns = m.nslot[c];
  const TV g = TV(m.gamma);
  // software pipeline over the slots: the column of slot t+2 and the
  // gathered x of slot t+1 are in flight while slot t is applied
  const int* __restrict__ sc = m.scol + (size_t)base * 32 + lane;
  int colA = ns > 0 ? sc[0] : 0;
  int colB = ns > 1 ? sc[32] : 0;
  TV xn[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) xn[k] = ns > 0 ? x[5 * (size_t)colA + k] : TV(0);
#pragma unroll UNR
  for (int t = 0; t < ns; ++t) {
    const int col = colA;
    TV xj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xj[k] = xn[k];
    colA = colB;
    if (t + 2 < ns) colB = sc[(t + 2) * 32];
    if (t + 1 < ns)
#pragma unroll
      for (int k = 0; k < 5; ++k) xn[k] = x[5 * (size_t)colA + k];
    SlotBlock<TB> Bk;
    Bk.load(blk, base + t, lane);
    add_slot<1>(Bk, g, xj, acc, part, (t & 1) || t == ns - 1);
    if (m.vjslot) vj_sub<TB>(m, base + t, lane, col, xj, acc);
  }
  if (m.nInst > 1 && hb_in_zone(m, c)) {
    const int J = c / m.Nc, cl = c - J * m.Nc;
    const double Vc = m.V[c];
    for (int K = 0; K < m.nInst; ++K) {
      if (K == J) continue;
      const TV d = TV(Vc * m.Dhb[J * m.nInst + K]);
      const TV* xk = x + 5 * ((size_t)K * m.Nc + cl);
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] += d * xk[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) w[5 * c + k] = acc[k];
}

template <typename TB, typename TV, int MINB = 1, int UNR = 1>
__global__ void __launch_bounds__(128, MINB) k_op_level1(DevMesh m, const TB* __restrict__ blk, const TB* __restrict__ dg,
                                                   const TB* __restrict__ rD, const TV* __restrict__ x,
                                                   TV* __restrict__ w, const int* __restrict__ cells, int start,
                                                   int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int c = cells ? cells[start + i] : start + i;
  const int s = c >> 5, lane = c & 31;
  TV xc[5], acc[5], part[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 5; ++k) xc[k] = x[5 * (size_t)c + k];
  const TB* D = dg + (size_t)s * 25 * 32 + lane;
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    TV a = TV(0);
#pragma unroll
    for (int j = 0; j < 5; ++j) a += TV(D[(5 * r + j) * 32]) * xc[j];
    acc[r] = a;
  }
  const int base = m.slot_base[s];
  const int ns = m.nslot[c];  // all lower: these rows have no upper neighbours
  const TV g = TV(m.gamma);
#pragma unroll UNR
  for (int t = 0; t < ns; ++t) {
    const int col = m.scol[(base + t) * 32 + lane];
    const TV rj = TV(rD[col]);
    // the product's x_j and the sweep's rD w_j meet the same block: one product
    TV xj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xj[k] = x[5 * (size_t)col + k] - rj * w[5 * col + k];
    SlotBlock<TB> Bk;
    Bk.load(blk, base + t, lane);
    add_slot<1>(Bk, g, xj, acc, part, (t & 1) || t == ns - 1);
    if (m.vjslot) vj_sub<TB>(m, base + t, lane, col, xj, acc);
  }
  if (m.nInst > 1 && hb_in_zone(m, c)) {
    const int J = c / m.Nc, cl = c - J * m.Nc;
    const double Vc = m.V[c];
    for (int K = 0; K < m.nInst; ++K) {
      if (K == J) continue;
      const TV d = TV(Vc * m.Dhb[J * m.nInst + K]);
      const TV* xk = x + 5 * ((size_t)K * m.Nc + cl);
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] += d * xk[k];
    }
  }
  const TV rc = TV(rD[c]);
#pragma unroll
  for (int k = 0; k < 5; ++k) w[5 * c + k] = rc * acc[k];
}

// ------------------------------------------------------------------ LU-SGS
// SCALE: also apply the reverse step of a row without upper neighbours
// (delta = rD * r'), fusing the last forward level with the first reverse one.
template <typename TB, typename TV, bool SCALE = false>
__device__ __forceinline__ void lusgs_fwd_row(const DevMesh& m, const TB* __restrict__ blk, const TB* __restrict__ rD,
                                              TV* __restrict__ r, int c) {
  const int s = c >> 5, lane = c & 31;
  const int base = m.slot_base[s];
  const int nl = m.nlow[c];
  TV acc[5], part[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 5; ++k) acc[k] = r[5 * c + k];
  const TV g = TV(m.gamma);
#pragma unroll 1
  for (int t = 0; t < nl; ++t) {
    const int col = m.scol[(base + t) * 32 + lane];
    const TV rj = TV(rD[col]);
    TV dj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) dj[k] = rj * r[5 * col + k];
    SlotBlock<TB> Bk;
    Bk.load(blk, base + t, lane);
    add_slot<-1>(Bk, g, dj, acc, part, (t & 1) || t == nl - 1);
    if (m.vjslot) vj_sub<TB, -1>(m, base + t, lane, col, dj, acc);
  }
  if (SCALE) {
    const TV rc = TV(rD[c]);
#pragma unroll
    for (int k = 0; k < 5; ++k) r[5 * c + k] = rc * acc[k];
  } else {
#pragma unroll
    for (int k = 0; k < 5; ++k) r[5 * c + k] = acc[k];
  }
}

template <typename TB, typename TV>
__device__ __forceinline__ void lusgs_rev_row(const DevMesh& m, const TB* __restrict__ blk, const TB* __restrict__ rD,
                                              TV* __restrict__ r, int c) {
  const int s = c >> 5, lane = c & 31;
  const int base = m.slot_base[s];
  const int nl = m.nlow[c], ns = m.nslot[c];
  TV acc[5], part[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 5; ++k) acc[k] = r[5 * c + k];
  // two slots in flight: their column loads and the dependent gathers overlap
  // (2% on the reverse sweep; a deeper software pipeline with the next slot's
  // column and deltas loaded ahead measured 11% slower)
  const TV g = TV(m.gamma);
  auto slot = [&](int t, bool flush) {
    const int col = m.scol[(base + t) * 32 + lane];
    TV dj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) dj[k] = r[5 * col + k];
    SlotBlock<TB> Bk;
    Bk.load(blk, base + t, lane);
    add_slot<-1>(Bk, g, dj, acc, part, flush);
    if (m.vjslot) vj_sub<TB, -1>(m, base + t, lane, col, dj, acc);
  };
  if constexpr (sizeof(TB) == 8) {
    int t = ns - 1;
    for (; t > nl; t -= 2) {  // flushed at compile time: an addition costs its cycles where predicated off too
      slot(t, false);
      slot(t - 1, true);
    }
    if (t == nl) slot(t, true);
  } else {
#pragma unroll 2
    for (int t = ns - 1; t >= nl; --t) slot(t, false);
  }
  const TV rc = TV(rD[c]);
#pragma unroll
  for (int k = 0; k < 5; ++k) r[5 * c + k] = rc * acc[k];
}

// Two rows of one reverse level in one thread: their slot loops run in
// lockstep, so the column index, block words and gathered neighbour rows of
// both are in flight together (a level's rows never read each other).  Each
// row's arithmetic is that of lusgs_rev_row: slots from the last down to the
// first upper one, acc -= B r_col, then the scaling by rD.
template <typename TB, typename TV>
__device__ __forceinline__ void lusgs_rev_row2(const DevMesh& m, const TB* __restrict__ blk,
                                               const TB* __restrict__ rD, TV* __restrict__ r, int c0, int c1) {
  const int l0 = c0 & 31, l1 = c1 & 31;
  const int b0 = m.slot_base[c0 >> 5], b1 = m.slot_base[c1 >> 5];
  const int nl0 = m.nlow[c0], nl1 = m.nlow[c1];
  int t0 = m.nslot[c0] - 1, t1 = m.nslot[c1] - 1;
  TV a0[5], a1[5], p0[5] = {0, 0, 0, 0, 0}, p1[5] = {0, 0, 0, 0, 0};
  bool odd = false;  // every second slot of the two rows
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    a0[k] = r[5 * c0 + k];
    a1[k] = r[5 * c1 + k];
  }
  const TV g = TV(m.gamma);
#pragma unroll 1
  for (; t0 >= nl0 || t1 >= nl1; --t0, --t1, odd = !odd) {
    const bool v0 = t0 >= nl0, v1 = t1 >= nl1;
    const int col0 = v0 ? m.scol[(b0 + t0) * 32 + l0] : c0;
    const int col1 = v1 ? m.scol[(b1 + t1) * 32 + l1] : c1;
    TV d0[5], d1[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      d0[k] = r[5 * col0 + k];
      d1[k] = r[5 * col1 + k];
    }
    SlotBlock<TB> B0, B1;
    if (v0) B0.load(blk, b0 + t0, l0);
    if (v1) B1.load(blk, b1 + t1, l1);
    if (v0) {
      add_slot<-1>(B0, g, d0, a0, p0, odd || t0 == nl0);
      if (m.vjslot) vj_sub<TB, -1>(m, b0 + t0, l0, col0, d0, a0);
    }
    if (v1) {
      add_slot<-1>(B1, g, d1, a1, p1, odd || t1 == nl1);
      if (m.vjslot) vj_sub<TB, -1>(m, b1 + t1, l1, col1, d1, a1);
    }
  }
  const TV rc0 = TV(rD[c0]), rc1 = TV(rD[c1]);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    r[5 * c0 + k] = rc0 * a0[k];
    r[5 * c1 + k] = rc1 * a1[k];
  }
}

// reverse level with two rows per thread: rows i and i + ceil(count/2)
template <typename TB, typename TV>
__global__ void __launch_bounds__(128) k_lusgs_rev2(DevMesh m, const TB* __restrict__ blk, const TB* __restrict__ rD,
                                                    TV* __restrict__ r, const int* __restrict__ cells, int start,
                                                    int count) {
  const int half = (count + 1) >> 1;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= half) return;
  const int c0 = cells ? cells[start + i] : start + i;
  if (i + half < count)
    lusgs_rev_row2<TB, TV>(m, blk, rD, r, c0, cells ? cells[start + i + half] : start + i + half);
  else
    lusgs_rev_row<TB, TV>(m, blk, rD, r, c0);
}

// one launch per level: cells = level list (nullptr when the level is the
// contiguous range [start, start+count))
// MODE 0: forward row, 1: reverse row, 2: forward row + reverse scaling
template <typename TB, typename TV, int MODE>
__global__ void __launch_bounds__(128) k_lusgs_level(DevMesh m, const TB* __restrict__ blk,
                                                     const TB* __restrict__ rD, TV* __restrict__ r,
                                                     const int* __restrict__ cells, int start, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int c = cells ? cells[start + i] : start + i;
  if (MODE == 0)
    lusgs_fwd_row<TB, TV>(m, blk, rD, r, c);
  else if (MODE == 1)
    lusgs_rev_row<TB, TV>(m, blk, rD, r, c);
  else
    lusgs_fwd_row<TB, TV, true>(m, blk, rD, r, c);
}

// ------------------------------------------------- FP64 rows on five lanes
// The FP64 products of few rows.  A warp's FP64 instruction holds its scheduler
// for 64 cycles, so a row per thread costs a warp 190 x 64 cycles for a product
// with six neighbours however few warps there are, while most of the 608
// schedulers idle.  Here five lanes share a row, one component each, six rows
// to a warp: 38 instructions per warp, in the same order per component.
// A row costs 7% more of the pipe in all, so the row-per-thread kernels stay for
// many rows.  By events around a launch (5 us of them), a row per thread against
// five lanes, product / second level / reverse: 5k rows 13.6 : 10.1 / 16.3 : 10.6
// / 16.3 : 10.5 us, 23.3k 19.0 : 14.9 / 21.4 : 16.7 / 20.8 : 14.9, 31.7k 20.2 :
// 18.9 / 23.4 : 22.6 / 22.3 : 19.2; from 39k rows (two full warps per scheduler)
// on neither way is ahead at every size, within 5% on average.
// ROWS_PRODUCT: w = A x (k_spmv, k_op_level0); ROWS_LEVEL1: k_op_level1;
// ROWS_REVERSE: the reverse sweep of a level, w in place (k_lusgs_level MODE 1).
enum { ROWS_PRODUCT, ROWS_LEVEL1, ROWS_REVERSE };
constexpr int ROWS5_WARP = 6;
constexpr int ROWS5_THREADS = 64;
constexpr int ROWS5_LIMIT = 36000;

template <int MODE>
__global__ void __launch_bounds__(ROWS5_THREADS) k_rows5(DevMesh m, const double* __restrict__ blk,
                                                         const double* __restrict__ dg,
                                                         const double* __restrict__ rD, const double* x, double* w,
                                                         const int* __restrict__ cells, int start, int count) {
  const int l = threadIdx.x & 31, r = l / 5, i = l - 5 * r;  // lanes 30, 31: idle
  const int row = (int)((blockIdx.x * ROWS5_THREADS + threadIdx.x) >> 5) * ROWS5_WARP + r;
  const bool on = r < ROWS5_WARP && row < count;
  const int c = on ? (cells ? cells[start + row] : start + row) : 0;
  const int lane = c & 31, base = m.slot_base[c >> 5];
  const int first = MODE == ROWS_REVERSE && on ? m.nlow[c] : 0, ns = on ? m.nslot[c] : 0;
  double acc = 0.0, part = 0.0;
  if (MODE == ROWS_REVERSE) {
    if (on) acc = w[5 * (size_t)c + i];
  } else if (on) {
    const double* D = dg + ((size_t)(c >> 5) * 25 + 5 * i) * 32 + lane;
#pragma unroll
    for (int j = 0; j < 5; ++j) acc += D[j * 32] * x[5 * (size_t)c + j];
  }
  const int trips = __reduce_max_sync(0xffffffffu, ns - first);
#pragma unroll 2
  for (int q = 0; q < trips; ++q) {
    const bool in = q < ns - first;
    const int t = MODE == ROWS_REVERSE ? ns - 1 - q : q;
    double B[5], xj[5], d = 0.0;
    int col = 0;
    if (in) {
      col = m.scol[(base + t) * 32 + lane];
      const double* bp = blk + ((size_t)(base + t) * 25 + 5 * i) * 32 + lane;
#pragma unroll
      for (int j = 0; j < 5; ++j) B[j] = bp[j * 32];
      if (MODE == ROWS_LEVEL1) {  // the product's x_j and the sweep's rD w_j meet the same block
        d = x[5 * (size_t)col + i] - rD[col] * w[5 * (size_t)col + i];
      } else {
        const double* from = MODE == ROWS_REVERSE ? w : x;
#pragma unroll
        for (int j = 0; j < 5; ++j) xj[j] = from[5 * (size_t)col + j];
      }
    }
    if (MODE == ROWS_LEVEL1)
#pragma unroll
      for (int j = 0; j < 5; ++j) xj[j] = __shfl_sync(0xffffffffu, d, min(5 * r, 25) + j);
    if (in) {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        if (MODE == ROWS_REVERSE) xj[j] = -xj[j];
        part += B[j] * xj[j];
      }
      if (m.vjslot) {
        double y[5] = {0, 0, 0, 0, 0};
        vj_sub<double>(m, base + t, lane, col, xj, y);
#pragma unroll
        for (int j = 0; j < 5; ++j)
          if (j == i) acc += y[j];
      }
    }
    if ((q & 1) || q == trips - 1) {  // as add_slot
      acc += part;
      part = 0.0;
    }
  }
  if (!on) return;
  if (MODE != ROWS_REVERSE && m.nInst > 1 && hb_in_zone(m, c)) {
    const int J = c / m.Nc, cl = c - J * m.Nc;
    const double Vc = m.V[c];
    for (int K = 0; K < m.nInst; ++K) {
      if (K == J) continue;
      acc += Vc * m.Dhb[J * m.nInst + K] * x[5 * ((size_t)K * m.Nc + cl) + i];
    }
  }
  w[5 * (size_t)c + i] = MODE == ROWS_PRODUCT ? acc : rD[c] * acc;
}

template <int MODE>
static bool rows5(Handle& h, int kind, const double* blk, const double* dg, const double* rD, const double* x, double* w,
                  const int* cells, int start, int count) {
  if (count > ROWS5_LIMIT) return false;
  const int perBlock = ROWS5_WARP * ROWS5_THREADS / 32;
  ICS_LAUNCH(h, kind, k_rows5<MODE><<<grid_for(count, perBlock), ROWS5_THREADS, 0, h.stream>>>(h.m, blk, dg, rD, x, w, cells,
                                                                                              start, count));
  return true;
}

// ----------------------------------------------- sync-free LU-SGS sweeps
// One launch per sweep for schedules with many levels (RCM / natural
// numbering).  A resident set of warps draws consecutive tickets; ticket t
// holds rows order[32 t .. 32 t + 31], the levels one after the other and
// each padded to whole tickets (-1), so a row only ever waits for rows of
// smaller tickets -- drawn earlier by warps that are resident or done and
// that never wait for a later one -- and never for a lane of its own warp:
// no deadlock.  The sweep writes its rows into a padded output array (8 words
// per row, 32 B for FP32) that starts filled with a sentinel (all bits set: a
// NaN with the sign bit, which GPU arithmetic does not produce from finite
// operands and which a row never publishes),
// and a row's result words are their own done flags: a row polls its
// neighbours' five words with relaxed loads until none is the sentinel.  One
// L2 round trip per poll brings both the readiness and the values, the writer
// needs no fence, and the polls of all prefetched neighbours are issued
// together.  Per row the neighbours are subtracted in the order of
// lusgs_fwd_row / lusgs_rev_row.  A wait that
// exceeds the bound sets status bit 8, publishes zeros (so that its
// dependents do not wait in turn) and goes on; waiting rows that see bit 8
// give up too (the host reports ICS_ERR_TIMEOUT).
constexpr int SWEEP_SPIN_LIMIT = 1 << 22;
constexpr int SWEEP_PAD = 8;  // words per row of the sweep outputs
constexpr int SWEEP_THREADS = 32;  // one warp per block
// rows a warp takes at once (sweep_row16 / sweep_row4)
template <typename TB, typename TV>
constexpr int sweep_rows = sizeof(TB) == 8 && sizeof(TV) == 8 ? 2 : 8;

__device__ __forceinline__ void ld_relaxed5(const float* p, float* v) {
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "l"(p)
               : "memory");
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v[4]) : "l"(p + 4) : "memory");
}
__device__ __forceinline__ void ld_relaxed5(const double* p, double* v) {
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p) : "memory");
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "l"(p + 2) : "memory");
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v[4]) : "l"(p + 4) : "memory");
}
__device__ __forceinline__ void st_relaxed5(float* p, const float* v) {
  asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3])
               : "memory");
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p + 4), "f"(v[4]) : "memory");
}
__device__ __forceinline__ void st_relaxed5(double* p, const double* v) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v[0]), "d"(v[1]) : "memory");
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p + 2), "d"(v[2]), "d"(v[3]) : "memory");
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p + 4), "d"(v[4]) : "memory");
}
__device__ __forceinline__ bool sweep_word_set(float v) { return __float_as_uint(v) != 0xffffffffu; }
__device__ __forceinline__ bool sweep_word_set(double v) {
  return (unsigned long long)__double_as_longlong(v) != ~0ull;
}
// a result that is the sentinel itself (a NaN of that payload in the input)
// is published as the canonical NaN, so that its dependents do not wait
__device__ __forceinline__ float sweep_word(float v) { return sweep_word_set(v) ? v : __uint_as_float(0x7fffffffu); }
__device__ __forceinline__ double sweep_word(double v) {
  return sweep_word_set(v) ? v : __longlong_as_double(0x7fffffffffffffffLL);
}
template <typename TV>
__device__ __forceinline__ bool sweep_ready(const TV* v) {
  return sweep_word_set(v[0]) && sweep_word_set(v[1]) && sweep_word_set(v[2]) && sweep_word_set(v[3]) &&
         sweep_word_set(v[4]);
}

// FWD: in = the right-hand side r (5 words per row), out = the forward
// result; !FWD: in = the forward result (padded), out = the reverse result,
// also written to r (5 words per row).  `out` holds the sentinel on entry.
//
// FP64 rows, 16 lanes each (two rows per warp): lane (p, i) = (lane / 5, lane
// % 5) of a row handles component i of its p-th neighbour of three, so the
// three neighbours are polled, scaled and multiplied at once.  GB300 issues a
// warp's FP64 instruction over 64 cycles of its scheduler whatever
// lanes are active, so a row costs its count of instructions: 10 here against
// 105 with one row per lane.  The sums keep the order of lusgs_fwd_row /
// lusgs_rev_row.
template <typename TB, bool FWD>
__device__ __forceinline__ void sweep_row16(const DevMesh& m, const TB* __restrict__ blk, const TB* __restrict__ rD,
                                            const double* in, double* out, double* r, int c, int* status,
                                            int spin_limit) {
  const unsigned half = 0xffffu << (threadIdx.x & 16);
  const int l16 = threadIdx.x & 15;
  const int p = l16 / 5, i = l16 - 5 * p;  // lane 15: idle (p == 3)
  const bool row = c >= 0;
  int sb = 0, nl = 0, nn = 0, ns = 0, lane = 0;
  double acc = 0.0, rc = 0.0;
  if (row) {
    const int s = c >> 5;
    lane = c & 31;
    sb = m.slot_base[s];
    nl = m.nlow[c];
    ns = m.nslot[c];
    nn = FWD ? nl : ns - nl;
    if (p == 0) acc = FWD ? __ldcg(in + 5 * (size_t)c + i) : __ldcg(in + SWEEP_PAD * (size_t)c + i);
    if (!FWD) rc = double(rD[c]);
  }
  for (int q0 = 0; __any_sync(half, q0 < nn); q0 += 3) {
    const int q = q0 + p;
    const bool on = p < 3 && q < nn;
    double B[5], rj = 1.0;
    int col = 0, t = 0;
    if (on) {
      t = FWD ? q : ns - 1 - q;
      col = m.scol[(sb + t) * 32 + lane];
      const double* bp = (const double*)blk + ((size_t)(sb + t) * 25 + 5 * i) * 32 + lane;
#pragma unroll
      for (int j = 0; j < 5; ++j) B[j] = bp[j * 32];
      if (FWD) rj = double(rD[col]);
    }
    // poll this lane's word; the lanes of a half-warp go on together
    double v = 0.0;
    bool ready = !on;
    int it = 0;
    while (true) {
      if (!ready) {
        asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(out + SWEEP_PAD * (size_t)col + i) : "memory");
        ready = sweep_word_set(v);
      }
      if (__all_sync(half, ready)) break;
      ++it;
      bool stop = it > spin_limit;
      if (stop && l16 == 0) atomicOr(status, 8);
      if ((it & 63) == 0) stop = stop || (ld_relaxed_int(status) & 8);
      if (__any_sync(half, stop)) {
        if (p == 0) {
          const double z = 0.0;
          asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(out + SWEEP_PAD * (size_t)c + i), "d"(z) : "memory");
        }
        return;
      }
    }
    const double d = FWD ? rj * v : v;
    double y = 0.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const double dj = __shfl_sync(half, d, 5 * p + j, 16);
      if (on) y += B[j] * dj;
    }
    if (m.vjslot) {
      // the non-LF viscous part needs the neighbour's five words in one lane
      double x5[5], y5[5] = {0, 0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 5; ++j) x5[j] = __shfl_sync(half, d, 5 * p + j, 16);
      if (on) {
        vj_sub<TB>(m, sb + t, lane, col, x5, y5);
#pragma unroll
        for (int j = 0; j < 5; ++j)
          if (j == i) y += y5[j];
      }
    }
    const double y1 = __shfl_sync(half, y, 5 + i, 16), y2 = __shfl_sync(half, y, (10 + i) & 15, 16);
    acc -= y;
    if (q0 + 1 < nn) acc -= y1;
    if (q0 + 2 < nn) acc -= y2;
  }
  if (row && p == 0) {
    if (!FWD) {
      acc = rc * acc;
      r[5 * (size_t)c + i] = acc;
    }
    acc = sweep_word(acc);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(out + SWEEP_PAD * (size_t)c + i), "d"(acc) : "memory");
  }
}

// Rows with FP32 blocks, 4 lanes each (eight rows per warp): lane p of a row polls,
// scales and multiplies its p-th neighbour of three, lane 0 subtracts the
// products in the order of lusgs_fwd_row / lusgs_rev_row.  A level costs the
// L2 path of its results and the row's dependent instructions, so fewer words
// per poll of a warp (8 rows x 3 neighbours) and one block product after the
// other's on its own lane shorten it: 0.86 us a level on a 227k-cell RCM
// box (181 levels), 1.5 with one row per lane.  A warp's rows go on together
// (they are of one level, and none waits for another).
template <typename TB, typename TV, bool FWD>
__device__ __forceinline__ void sweep_row4(const DevMesh& m, const TB* __restrict__ blk, const TB* __restrict__ rD,
                                           const TV* in, TV* out, TV* r, int c, int* status,
                                           int spin_limit) {
  const int p = threadIdx.x & 3;  // lane 3: idle
  const bool row = c >= 0;
  int sb = 0, nl = 0, nn = 0, ns = 0, lane = 0;
  TV acc[5] = {0, 0, 0, 0, 0}, rc = TV(0);
  if (row) {
    const int s = c >> 5;
    lane = c & 31;
    sb = m.slot_base[s];
    nl = m.nlow[c];
    ns = m.nslot[c];
    nn = FWD ? nl : ns - nl;
    if (p == 0) {
#pragma unroll
      for (int k = 0; k < 5; ++k) acc[k] = FWD ? __ldcg(in + 5 * (size_t)c + k) : __ldcg(in + SWEEP_PAD * (size_t)c + k);
      if (!FWD) rc = TV(rD[c]);
    }
  }
  const TV g = TV(m.gamma);
  for (int q0 = 0; __any_sync(0xffffffffu, q0 < nn); q0 += 3) {
    const int q = q0 + p;
    const bool on = p < 3 && q < nn;
    SlotBlock<TB> B = {};
    TV rj = TV(1), v[5] = {0, 0, 0, 0, 0}, y[5] = {0, 0, 0, 0, 0};
    int col = 0, t = 0;
    if (on) {
      t = FWD ? q : ns - 1 - q;
      col = m.scol[(sb + t) * 32 + lane];
      B.load(blk, sb + t, lane);
      if (FWD) rj = TV(rD[col]);
    }
    // the terms of the product that do not wait for the neighbour, made before
    // the wait (the empty statement keeps them there)
    typename SlotBlock<TB>::template Terms<TV> terms(g, B.w);
    if constexpr (sizeof(TV) == 4) asm volatile("" : "+f"(terms.th), "+f"(terms.a1), "+f"(terms.pu));
    bool ready = !on;
    int it = 0;
    while (true) {
      if (!ready) {
        ld_relaxed5(out + SWEEP_PAD * (size_t)col, v);
        ready = sweep_ready(v);
      }
      if (__all_sync(0xffffffffu, ready)) break;
      ++it;
      bool stop = it > spin_limit;
      if (stop && threadIdx.x == 0) atomicOr(status, 8);
      if ((it & 63) == 0) stop = stop || (ld_relaxed_int(status) & 8);
      if (__any_sync(0xffffffffu, stop)) {
        const TV z[5] = {0, 0, 0, 0, 0};
        if (row && p == 0) st_relaxed5(out + SWEEP_PAD * (size_t)c, z);
        return;
      }
    }
    if (on) {
      TV d[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) d[k] = FWD ? rj * v[k] : v[k];
      terms.apply(g, d, y);
      if (m.vjslot) vj_sub<TB>(m, sb + t, lane, col, d, y);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {  // an idle lane's product is zero
      const TV y1 = __shfl_down_sync(0xffffffffu, y[k], 1, 4), y2 = __shfl_down_sync(0xffffffffu, y[k], 2, 4);
      acc[k] = ((acc[k] - y[k]) - y1) - y2;
    }
  }
  if (row && p == 0) {
    TV z[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      if (!FWD) acc[k] = rc * acc[k];
      z[k] = sweep_word(acc[k]);
    }
    st_relaxed5(out + SWEEP_PAD * (size_t)c, z);
    if (!FWD)
#pragma unroll
      for (int k = 0; k < 5; ++k) r[5 * (size_t)c + k] = acc[k];
  }
}

template <typename TB, typename TV, bool FWD>
__global__ void __launch_bounds__(SWEEP_THREADS) k_lusgs_sweep(DevMesh m, const TB* __restrict__ blk,
                                                     const TB* __restrict__ rD, const TV* in, TV* out, TV* r,
                                                     const int* __restrict__ order, int tickets,
                                                     unsigned int* ticket, int* status, int spin_limit) {
  constexpr int ROWS = sweep_rows<TB, TV>;
  const int total = tickets * (SWEEP_TICKET / ROWS);
  while (true) {
    int t = 0;
    if (threadIdx.x == 0) t = (int)atomicAdd(ticket, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= total) return;
    const int c = order[t * ROWS + threadIdx.x / (32 / ROWS)];
    if constexpr (ROWS == 2)
      sweep_row16<TB, FWD>(m, blk, rD, in, out, r, c, status, spin_limit);
    else
      sweep_row4<TB, TV, FWD>(m, blk, rD, in, out, r, c, status, spin_limit);
    __syncwarp();
  }
}

template <typename TB, typename TV>
__global__ void k_jacobi_apply(int N, const TB* __restrict__ inv, TV* __restrict__ r) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  const int s = c >> 5, lane = c & 31;
  const TB* D = inv + (size_t)s * 25 * 32 + lane;
  TV x[5], z[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) x[k] = r[5 * c + k];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    TV a = TV(0);
#pragma unroll
    for (int j = 0; j < 5; ++j) a += TV(D[(5 * i + j) * 32]) * x[j];
    z[i] = a;
  }
#pragma unroll
  for (int k = 0; k < 5; ++k) r[5 * c + k] = z[k];
}

// ------------------------------------------------------------ vector kernels
template <typename TS, typename TD>
__global__ void k_cast(long n, const TS* __restrict__ a, TD* __restrict__ b) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    if constexpr (sizeof(TS) == 4)
      b[i] = widen(a[i]);
    else
      b[i] = convert<TD>(a[i]);
  }
}

__device__ __forceinline__ void addmul16(float4& a, float y, const float4& v) {
  a.x += y * v.x;
  a.y += y * v.y;
  a.z += y * v.z;
  a.w += y * v.w;
}
__device__ __forceinline__ void addmul16(double2& a, double y, const double2& v) {
  a.x += y * v.x;
  a.y += y * v.y;
}

// the last direction's Givens rotation, then H y = bh (one warp)
__global__ void __launch_bounds__(32) k_backsub(KrylovScalars* ks, int m) {
  if (ks->status) return;
  if (threadIdx.x == 0) dev_hess(ks, m - 1, m);
  __syncwarp();
  back_substitute(ks->H, ks->bh, ks->y, m);
}

template <typename TV>
__global__ void __launch_bounds__(RB) k_xupdate(long n, TV* __restrict__ x, const TV* __restrict__ V,
                                                const KrylovScalars* __restrict__ ks, int m, long vstride) {
  __shared__ TV y[MAX_DIRS];  // converted once, not per element
  if (ks->status) return;
  if ((int)threadIdx.x < m) y[threadIdx.x] = convert<TV>(ks->y[threadIdx.x]);
  __syncthreads();
  using VT = typename V16<TV>::T;
  constexpr int L = V16<TV>::n;
  const long nv = n / L;
  const long stride = (long)gridDim.x * blockDim.x;
  VT* x4 = reinterpret_cast<VT*>(x);
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < nv; q += stride) {
    VT a = x4[q];
#pragma unroll 4
    for (int i = 0; i < m; ++i) addmul16(a, y[i], reinterpret_cast<const VT*>(V + (size_t)i * vstride)[q]);
    x4[q] = a;
  }
  for (long q = nv * L + blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += stride) {
    TV a = x[q];
    for (int i = 0; i < m; ++i) a += y[i] * V[(size_t)i * vstride + q];
    x[q] = a;
  }
}

// Per-instance reductions: blockIdx.y is the instance, whose Nc cells start at
// y*Nc; each instance folds its own partials and counter into out + y*NV.
#define ICS_INSTANCE_RANGE(Nc)                                     \
  const int inst_ = blockIdx.y;                                    \
  const int cend_ = (inst_ + 1) * (Nc);                            \
  partials += (size_t)inst_ * gridDim.x * NV_;                     \
  counter += inst_;                                                \
  out += inst_ * NV_;

// r = b - t, per-equation L1 sums of r (rho, rhoUx, rhoUy, rhoUz, rhoE)
template <typename TV>
__global__ void __launch_bounds__(RB) k_resid(int Nc, const double* __restrict__ b, const TV* __restrict__ t,
                                              TV* __restrict__ r, double* __restrict__ partials,
                                              unsigned int* __restrict__ counter, double* __restrict__ out) {
  constexpr int NV_ = 5;
  ICS_INSTANCE_RANGE(Nc)
  double acc[5] = {0, 0, 0, 0, 0};
  for (int c = inst_ * Nc + blockIdx.x * blockDim.x + threadIdx.x; c < cend_; c += gridDim.x * blockDim.x) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const TV v = convert<TV>(b[5 * c + k]) - t[5 * c + k];
      r[5 * c + k] = v;
      acc[k] += fabs(widen(v));
    }
  }
  reduce_finish<5>(acc, partials, counter, out);
}

// sums of |b_k| (initial residual) and the norm factors
template <typename TV>
__global__ void __launch_bounds__(RB) k_normfac(int Nc, const double* __restrict__ b, const TV* __restrict__ t,
                                                double* __restrict__ partials, unsigned int* __restrict__ counter,
                                                double* __restrict__ out) {
  // out per instance: nf_rho, nf_rhoE, nf_rhoU, |b| rho, Ux, Uy, Uz, rhoE
  constexpr int NV_ = 8;
  ICS_INSTANCE_RANGE(Nc)
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int c = inst_ * Nc + blockIdx.x * blockDim.x + threadIdx.x; c < cend_; c += gridDim.x * blockDim.x) {
    const double t0 = widen(t[5 * c]), t4 = widen(t[5 * c + 4]);
    const double t1 = widen(t[5 * c + 1]), t2 = widen(t[5 * c + 2]), t3 = widen(t[5 * c + 3]);
    const double b0 = b[5 * c], b1 = b[5 * c + 1], b2 = b[5 * c + 2], b3 = b[5 * c + 3], b4 = b[5 * c + 4];
    acc[0] += fabs(t0) + fabs(b0);
    acc[1] += fabs(t4) + fabs(b4);
    acc[2] += sqrt(t1 * t1 + t2 * t2 + t3 * t3) + sqrt(b1 * b1 + b2 * b2 + b3 * b3);
    acc[3] += fabs(b0);
    acc[4] += fabs(b1);
    acc[5] += fabs(b2);
    acc[6] += fabs(b3);
    acc[7] += fabs(b4);
  }
  reduce_finish<8>(acc, partials, counter, out);
}

// the averages of W per equation and instance (gAverage)
__global__ void __launch_bounds__(RB) k_wavg(int Nc, const double* __restrict__ W, double* __restrict__ partials,
                                             unsigned int* __restrict__ counter, double* __restrict__ out) {
  constexpr int NV_ = 5;
  ICS_INSTANCE_RANGE(Nc)
  double acc[5] = {0, 0, 0, 0, 0};
  for (int c = inst_ * Nc + blockIdx.x * blockDim.x + threadIdx.x; c < cend_; c += gridDim.x * blockDim.x)
#pragma unroll
    for (int k = 0; k < 5; ++k) acc[k] += W[5 * c + k];
  if (reduce_finish<5>(acc, partials, counter, out))
    for (int k = 0; k < 5; ++k) out[k] = out[k] / Nc;
}

template <typename TV>
__global__ void k_wmavg(int N, int Nc, const double* __restrict__ W, const KrylovScalars* __restrict__ ks,
                        TV* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  const double* avg = ks->avg + 5 * (c / Nc);
#pragma unroll
  for (int k = 0; k < 5; ++k) out[5 * c + k] = convert<TV>(W[5 * c + k] - avg[k]);
}

template <typename TV>
__global__ void k_to_dW(int N, const TV* __restrict__ x, double* __restrict__ dW, int s0, int s1, int s2) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= N) return;
  dW[5 * c] = widen(x[5 * c]);
  dW[5 * c + 1] = s0 == -1 ? 0.0 : widen(x[5 * c + 1]);
  dW[5 * c + 2] = s1 == -1 ? 0.0 : widen(x[5 * c + 2]);
  dW[5 * c + 3] = s2 == -1 ? 0.0 : widen(x[5 * c + 3]);
  dW[5 * c + 4] = widen(x[5 * c + 4]);
}

__global__ void __launch_bounds__(RB) k_sumsq(int N, const double* __restrict__ a, double* __restrict__ partials,
                                              unsigned int* __restrict__ counter, double* __restrict__ out) {
  double acc[1] = {0.0};
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) acc[0] += a[c];
  reduce_finish<1>(acc, partials, counter, out);
}

// -------------------------------------------------------------- dispatch
template <typename TB, typename TV>
static void spmv_t(Handle& h, const TV* x, TV* y) {
  bool split = false;
  if constexpr (sizeof(TB) == 8)
    split = rows5<ROWS_PRODUCT>(h, ICS_K_SPMV, (const double*)h.blk, (const double*)h.dg, nullptr, x, y, nullptr, 0, h.m.N);
  if (!split)
    ICS_LAUNCH(h, ICS_K_SPMV, k_spmv<TB, TV><<<grid_for(h.m.N, 128), 128, 0, h.stream>>>(h.m, (const TB*)h.blk, (const TB*)h.dg, x, y));
  if (h.m.ncrow > 0)
    ICS_LAUNCH(h, ICS_K_SPMV, k_cyc_mv<TB, TV><<<grid_for(h.m.ncrow, 128), 128, 0, h.stream>>>(h.m, (const TB*)h.cblk, x, y));
}


// one reverse level: one row per thread, or two (Handle::tuneRevRows)
template <typename TB, typename TV>
static void rev_level(Handle& h, const TB* blk, const TB* rD, TV* r, const int* cells, int start, int cnt) {
  if constexpr (sizeof(TB) == 8)
    if (rows5<ROWS_REVERSE>(h, ICS_K_LUSGS_REV, blk, nullptr, rD, nullptr, r, cells, start, cnt)) return;
  if (h.tuneRevRows == 2)
    ICS_LAUNCH(h, ICS_K_LUSGS_REV, k_lusgs_rev2<TB, TV><<<grid_for((cnt + 1) / 2, 128), 128, 0, h.stream>>>(
                                       h.m, blk, rD, r, cells, start, cnt));
  else
    ICS_LAUNCH(h, ICS_K_LUSGS_REV, k_lusgs_level<TB, TV, 1><<<grid_for(cnt, 128), 128, 0, h.stream>>>(
                                       h.m, blk, rD, r, cells, start, cnt));
}

// whether some reverse level runs the kernels that Handle::tuneRevRows chooses
// between: not with the sync-free sweeps, the chain scan or another
// preconditioner, nor where every level's rows are on five lanes each
template <typename TB>
static bool rev_rows_choice(const Handle& h) {
  const DevMesh& m = h.m;
  if (m.sw_fwd || h.cfg.c.preconditioner != ICS_PC_LUSGS) return false;
  for (int l = m.fuse_last ? 1 : 0; l < m.nrl; ++l)
    if (sizeof(TB) == 4 || m.rl_ptr[l + 1] - m.rl_ptr[l] > ROWS5_LIMIT) return true;
  return false;
}

// Resident warps of a sync-free sweep: a few levels' worth, so that the loads
// of the next levels' rows are in flight while a level is polled, and no more
// pollers than that.  Measured on a 227k-cell RCM box (181 levels): two rows
// per warp (FP64 blocks), one / two / four / eight levels 537 / 340 / 276 /
// 278 us per sweep; eight rows per warp, two / three / four / six / eight
// levels 235 / 186 / 165 / 157 / 157 us (1M cells in the natural order 531 /
// 450 / 443 / 427 / 438).
static int sweep_grid(const DevMesh& m, int tickets, int rows) {
  const long warps = (long)tickets * (SWEEP_TICKET / rows);
  const long g = std::min(std::max((rows == 2 ? 4 : 6) * warps / m.nfl, 152L), 152L * 32);
  return (int)std::min(g, warps);
}

template <typename TB, typename TV>
static void lusgs_t(Handle& h, TV* r, const TB* blkIn = nullptr, const TB* rDIn = nullptr) {
  const DevMesh& m = h.m;
  const TB* blk = blkIn ? blkIn : (const TB*)h.blk;
  const TB* rD = rDIn ? rDIn : (const TB*)h.rD;
  if (m.chain && !blkIn) {
    chain_sweeps(h, r);
    return;
  }
  // many levels: one sync-free launch per sweep
  if (m.sw_fwd) {
    cudaStream_t st = h.stream;
    int* status = &h.ks->status;
    TV* fwd = (TV*)m.sweep_pad;
    TV* rev = fwd + (size_t)SWEEP_PAD * m.N;
    const size_t padBytes = (size_t)SWEEP_PAD * m.N * sizeof(TV);
    ICS_CUDA(cudaMemsetAsync(fwd, 0xff, 2 * padBytes, st));  // the sentinel in both outputs
    ICS_CUDA(cudaMemsetAsync(m.sweep_ticket, 0, 2 * sizeof(unsigned int), st));
    const int grid = sweep_grid(m, m.nsw_fwd, sweep_rows<TB, TV>);
    const int spin = h.sweepProbe ? h.sweepProbe : SWEEP_SPIN_LIMIT;
    const int* fwdOrder = h.sweepProbe ? h.sweepProbeOrder : m.sw_fwd;
    ICS_LAUNCH(h, ICS_K_LUSGS_FWD, k_lusgs_sweep<TB, TV, true><<<grid, SWEEP_THREADS, 0, st>>>(
                                       m, blk, rD, r, fwd, nullptr, fwdOrder, m.nsw_fwd, m.sweep_ticket, status,
                                       spin));
    ICS_LAUNCH(h, ICS_K_LUSGS_REV, k_lusgs_sweep<TB, TV, false><<<grid, SWEEP_THREADS, 0, st>>>(
                                       m, blk, rD, fwd, rev, r, m.sw_rev, m.nsw_rev, m.sweep_ticket + 1, status,
                                       spin));
    return;
  }
  // One or two levels (colour-blocked numberings): a launch per level.
  // Forward level 0 has no lower neighbours (r' = r): skipped.  When the last
  // forward level holds exactly the rows of the first reverse level (rows
  // without upper neighbours, e.g. the last colour), the two are fused:
  // r' = r - L d*, then delta = rD r' in the same pass.
  for (int l = 0; l < m.nfl; ++l) {
    const bool last = l == m.nfl - 1;
    if (l == 0 && !(m.fuse_last && last)) continue;
    const int a = m.fl_ptr[l], cnt = m.fl_ptr[l + 1] - a;
    const bool contig = m.fl_cstart[l] >= 0;
    const int* cells = contig ? nullptr : m.fl_cells;
    const int start = contig ? m.fl_cstart[l] : a;
    if (m.fuse_last && last)
      ICS_LAUNCH(h, ICS_K_LUSGS_FWD, k_lusgs_level<TB, TV, 2><<<grid_for(cnt, 128), 128, 0, h.stream>>>(
                                         m, blk, rD, r, cells, start, cnt));
    else
      ICS_LAUNCH(h, ICS_K_LUSGS_FWD, k_lusgs_level<TB, TV, 0><<<grid_for(cnt, 128), 128, 0, h.stream>>>(
                                         m, blk, rD, r, cells, start, cnt));
  }
  for (int l = m.fuse_last ? 1 : 0; l < m.nrl; ++l) {
    const int a = m.rl_ptr[l], cnt = m.rl_ptr[l + 1] - a;
    const bool contig = m.rl_cstart[l] >= 0;
    rev_level<TB, TV>(h, blk, rD, r, contig ? nullptr : m.rl_cells, contig ? m.rl_cstart[l] : a, cnt);
  }
}

// w = M^-1 A x with M the LU-SGS preconditioner; true when the fused
// three-pass form applies (two levels, the second without upper neighbours)
template <typename TB, typename TV>
static bool fused_op_available(const Handle& h) {
  const DevMesh& m = h.m;
  // (the fused passes carry no cyclic couplings: those meshes take spmv_t)
  return h.tuneFused && h.cfg.c.preconditioner == ICS_PC_LUSGS && m.nfl == 2 && m.nrl == 2 && m.fuse_last &&
         m.ncyc == 0;
}

template <typename TB, typename TV>
static bool fused_op_t(Handle& h, const TV* x, TV* w) {
  const DevMesh& m = h.m;
  if (!fused_op_available<TB, TV>(h)) return false;
  const TB* blk = (const TB*)h.blk;
  const TB* dg = (const TB*)h.dg;
  const TB* rD = (const TB*)h.rD;
  auto level = [&](int l, const int** cells, int* start, int* cnt) {
    const int a = m.fl_ptr[l];
    *cnt = m.fl_ptr[l + 1] - a;
    const bool contig = m.fl_cstart[l] >= 0;
    *cells = contig ? nullptr : m.fl_cells;
    *start = contig ? m.fl_cstart[l] : a;
  };
  const int* c0;
  const int* c1;
  int s0, n0, s1, n1;
  level(0, &c0, &s0, &n0);
  level(1, &c1, &s1, &n1);
  // slot loops not unrolled; FP32: at least 8 blocks of 128 per SM (64
  // registers), with the factored slots 4-7% faster per pass than two slots
  // in flight or the compiler's register choice (72-80), and 10 or 12 blocks
  // (51 / 40 registers, the latter spilling) were not faster; FP64 would spill
  constexpr int OPB = sizeof(TB) == 4 ? 8 : 1;
  bool split0 = false, split1 = false;
  if constexpr (sizeof(TB) == 8) {
    split0 = n0 && rows5<ROWS_PRODUCT>(h, ICS_K_OP0, blk, dg, nullptr, x, w, c0, s0, n0);
    split1 = n1 && rows5<ROWS_LEVEL1>(h, ICS_K_OP1, blk, dg, rD, x, w, c1, s1, n1);
  }
  if (n0 && !split0)
    ICS_LAUNCH(h, ICS_K_OP0, k_op_level0<TB, TV, OPB, 1><<<grid_for(n0, 128), 128, 0, h.stream>>>(m, blk, dg, x, w, c0,
                                                                                                 s0, n0));
  if (n1 && !split1)
    ICS_LAUNCH(h, ICS_K_OP1, k_op_level1<TB, TV, OPB, 1><<<grid_for(n1, 128), 128, 0, h.stream>>>(m, blk, dg, rD, x, w,
                                                                                                 c1, s1, n1));
  // reverse level 1 = forward level 0 rows
  const int a = m.rl_ptr[1], cnt = m.rl_ptr[2] - a;
  const bool contig = m.rl_cstart[1] >= 0;
  if (cnt) rev_level<TB, TV>(h, blk, rD, w, contig ? nullptr : m.rl_cells, contig ? m.rl_cstart[1] : a, cnt);
  return true;
}

template <typename TB, typename TV>
static void precondition_t(Handle& h, TV* r) {
  if (h.cfg.c.preconditioner == ICS_PC_LUSGS)
    lusgs_t<TB, TV>(h, r);
  else if (h.cfg.c.preconditioner == ICS_PC_JACOBI)
    ICS_LAUNCH(h, ICS_K_JACOBI, k_jacobi_apply<TB, TV><<<grid_for(h.m.N, 128), 128, 0, h.stream>>>(h.m.N, (const TB*)h.dginv, r));
}

// One sync-free forward sweep over `order` (whole tickets) with a given wait
// bound; used to exercise the bounded waits (a row left out of the order
// never writes its result, so its dependents must give up and report).
template <typename TB, typename TV>
static void sweep_probe_t(Handle& h, const int* order, int tickets, int spin_limit) {
  const DevMesh& m = h.m;
  cudaStream_t st = h.stream;
  TV* fwd = (TV*)m.sweep_pad;
  ICS_CUDA(cudaMemsetAsync(fwd, 0xff, (size_t)SWEEP_PAD * m.N * sizeof(TV), st));
  ICS_CUDA(cudaMemsetAsync(m.sweep_ticket, 0, 2 * sizeof(unsigned int), st));
  ICS_CUDA(cudaMemsetAsync(h.kw, 0, 5ull * m.N * sizeof(TV), st));
  ICS_LAUNCH(h, ICS_K_LUSGS_FWD, k_lusgs_sweep<TB, TV, true><<<sweep_grid(m, tickets, sweep_rows<TB, TV>), SWEEP_THREADS, 0, st>>>(
                                     m, (const TB*)h.blk, (const TB*)h.rD, (const TV*)h.kw, fwd, nullptr, order,
                                     tickets, m.sweep_ticket, &h.ks->status, spin_limit));
  ICS_CUDA(cudaGetLastError());
}

// LU-SGS sweeps on an FP64 vector with the given off-diagonal slots (factored
// FP32 or 25-entry FP64 storage) and scalar diagonal: the preconditioner of
// the matrix-free Krylov solves (k_krylov.cu), which transposes the blocks
// for the adjoint system
void lusgs_with(Handle& h, const void* blk, const void* rD, bool fp32, double* r) {
  if (fp32)
    lusgs_t<float, double>(h, r, (const float*)blk, (const float*)rD);
  else
    lusgs_t<double, double>(h, r, (const double*)blk, (const double*)rD);
  ICS_CUDA(cudaGetLastError());
}

bool fused_operator(Handle& h, const void* x, void* w) {
  if (prec(h) == ICS_PREC_MIXED) return fused_op_t<float, float>(h, (const float*)x, (float*)w);
  return fused_op_t<double, double>(h, (const double*)x, (double*)w);
}

void sweep_probe(Handle& h, const int* order, int tickets, int spin_limit) {
  if (prec(h) == ICS_PREC_MIXED)
    sweep_probe_t<float, float>(h, order, tickets, spin_limit);
  else
    sweep_probe_t<double, double>(h, order, tickets, spin_limit);
}

void spmv(Handle& h, const void* x, void* y) {
  if (prec(h) == ICS_PREC_MIXED)
    spmv_t<float, float>(h, (const float*)x, (float*)y);
  else
    spmv_t<double, double>(h, (const double*)x, (double*)y);
  ICS_CUDA(cudaGetLastError());
}

int precondition(Handle& h, void* r) {
  if (prec(h) == ICS_PREC_MIXED)
    precondition_t<float, float>(h, (float*)r);
  else
    precondition_t<double, double>(h, (double*)r);
  ICS_CUDA(cudaGetLastError());
  return ICS_OK;
}

void to_vec(Handle& h, const double* src, void* dst) {
  const long n = 5L * h.m.N;
  if (prec(h) == ICS_PREC_MIXED)
    ICS_LAUNCH(h, ICS_K_VECTOR, k_cast<double, float><<<pass_grid(n), RB, 0, h.stream>>>(n, src, (float*)dst));
  else
    ICS_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDeviceToDevice, h.stream));
}

void from_vec(Handle& h, const void* src, double* dst) {
  const long n = 5L * h.m.N;
  if (prec(h) == ICS_PREC_MIXED)
    ICS_LAUNCH(h, ICS_K_VECTOR, k_cast<float, double><<<pass_grid(n), RB, 0, h.stream>>>(n, (const float*)src, dst));
  else
    ICS_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDeviceToDevice, h.stream));
}

// ----------------------------------------------------------------- GMRES
// residualsIO of the coupled system: initial and final L1 residuals per
// instance and equation, [5*J + k]
struct ResIO {
  std::vector<double> init, fin;
  int nIter = 0;
};

// coupledMatrix::solver::stop (coupledMatrixSolver.C:198-221) over every entry
static bool stop_test(const Handle& h, const ResIO& r) {
  const ics_config& c = h.cfg.c;
  if (r.nIter < c.min_iter) return false;
  double mx = -VGREAT, mrel = -VGREAT;
  for (double v : r.fin) mx = fmax(mx, v);
  for (int J = 0; J < h.m.nInst; ++J) {
    const double* in = &r.init[5 * J];
    const double* fi = &r.fin[5 * J];
    mrel = fmax(mrel, fi[0] / (in[0] + ROOTVSMALL));
    mrel = fmax(mrel, fi[4] / (in[4] + ROOTVSMALL));
    for (int k = 0; k < 3; ++k)
      if (h.m.solD[k] == 1) mrel = fmax(mrel, fi[1 + k] / (in[1 + k] + ROOTVSMALL));
  }
  return r.nIter >= c.max_iter || mx < c.tolerance || mrel < c.rel_tol;
}

// grid of the per-instance reductions: the instances share REDUCE_BLOCKS
static dim3 inst_grid(const Handle& h) {
  return dim3(std::max(1, std::min(REDUCE_BLOCKS / h.m.nInst, reduce_grid(h.m.Nc))), h.m.nInst);
}

// final L1 residuals from the per-instance sums in h.ksHost->res; false when
// any is not finite
static bool final_residuals(const Handle& h, const std::vector<double>& nf, ResIO& r) {
  bool finite = true;
  for (int J = 0; J < h.m.nInst; ++J) {
    const double* rs = h.ksHost->res + 5 * J;
    double* fi = &r.fin[5 * J];
    fi[0] = rs[0] / nf[3 * J];
    fi[4] = rs[4] / nf[3 * J + 1];
    for (int k = 0; k < 3; ++k) fi[1 + k] = h.m.solD[k] == -1 ? 0.0 : rs[1 + k] / nf[3 * J + 2];
    for (int k = 0; k < 5; ++k) finite = finite && std::isfinite(fi[k]);
  }
  return finite;
}

// Norm factors of coupledMatrixSolver (gmres.C:812-850): sum |A (W - avg W)| +
// |b| per equation (vector magnitude for rhoU), and the initial L1 residuals,
// each per instance (gAverage and gSum per field).
template <typename TB, typename TV>
static void norm_factors_t(Handle& h, std::vector<double>& nf, ResIO& r) {
  const int N = h.m.N, Nc = h.m.Nc, nI = h.m.nInst;
  cudaStream_t st = h.stream;
  KrylovScalars* ks = h.ks;
  TV* w = (TV*)h.kw;
  TV* t = (TV*)h.kt;
  const dim3 g = inst_grid(h);
  ICS_CUDA(cudaMemsetAsync(&ks->status, 0, sizeof(int), st));
  ICS_LAUNCH(h, ICS_K_VECTOR, k_wavg<<<g, RB, 0, st>>>(Nc, h.W, h.partials, h.counter, ks->avg));
  ICS_LAUNCH(h, ICS_K_VECTOR, k_wmavg<TV><<<grid_for(N, 256), 256, 0, st>>>(N, Nc, h.W, ks, w));
  spmv_t<TB, TV>(h, w, t);
  ICS_LAUNCH(h, ICS_K_VECTOR, k_normfac<TV><<<g, RB, 0, st>>>(Nc, h.src, t, h.partials, h.counter, ks->nfr));
  ICS_CUDA(cudaMemcpyAsync(h.ksHost->nfr, ks->nfr, 8 * nI * sizeof(double), cudaMemcpyDeviceToHost, st));
  ICS_CUDA(cudaStreamSynchronize(st));
  nf.assign(3 * nI, 0.0);
  r.init.assign(5 * nI, 0.0);
  r.nIter = 0;
  for (int J = 0; J < nI; ++J) {
    const double* q = h.ksHost->nfr + 8 * J;
    for (int k = 0; k < 3; ++k) nf[3 * J + k] = q[k] + VSMALL;
    double* in = &r.init[5 * J];
    in[0] = q[3] / nf[3 * J];
    in[1] = q[4] / nf[3 * J + 2];
    in[2] = q[5] / nf[3 * J + 2];
    in[3] = q[6] / nf[3 * J + 2];
    in[4] = q[7] / nf[3 * J + 1];
  }
  r.fin = r.init;
}

// x_new = D^-1 (b - (A - D) x_old): one block-Jacobi sweep (JacobiSmoother::smooth)
template <typename TB, typename TV>
__global__ void __launch_bounds__(128) k_jacobi_sweep(DevMesh m, const TB* __restrict__ blk,
                                                      const TB* __restrict__ inv, const double* __restrict__ b,
                                                      const TV* __restrict__ xo, TV* __restrict__ xn) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.N) return;
  const int s = c >> 5, lane = c & 31;
  TV acc[5] = {TV(0), TV(0), TV(0), TV(0), TV(0)}, part[5] = {0, 0, 0, 0, 0};
  const int base = m.slot_base[s], ns = m.nslot[c];
  const TV g = TV(m.gamma);
  for (int t = 0; t < ns; ++t) {
    const int col = m.scol[(base + t) * 32 + lane];
    TV xj[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xj[k] = xo[5 * col + k];
    SlotBlock<TB> Bk;
    Bk.load(blk, base + t, lane);
    add_slot<1>(Bk, g, xj, acc, part, (t & 1) || t == ns - 1);
    if (m.vjslot) vj_sub<TB>(m, base + t, lane, col, xj, acc);
  }
  TV r[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) r[k] = -(acc[k] - TV(b[5 * c + k]));
  const TB* D = inv + (size_t)s * 25 * 32 + lane;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    TV a = TV(0);
#pragma unroll
    for (int j = 0; j < 5; ++j) a += TV(D[(5 * i + j) * 32]) * r[j];
    xn[5 * c + i] = a;
  }
}

// smoothSolverCoupled::solveDelta (smoothSolverCoupled.C:369-515)
template <typename TB, typename TV>
static int smooth_t(Handle& h, ResIO& p) {
  const int N = h.m.N;
  const long n5 = 5L * N;
  cudaStream_t st = h.stream;
  KrylovScalars* ks = h.ks;
  std::vector<double> nf;
  norm_factors_t<TB, TV>(h, nf, p);
  TV* x = (TV*)h.kx;
  TV* y = (TV*)h.kb;
  TV* t = (TV*)h.kt;
  TV* r = (TV*)h.kw;
  ICS_CUDA(cudaMemsetAsync(x, 0, n5 * sizeof(TV), st));
  bool finite = true;
  do {
    for (int s = 0; s < h.cfg.c.n_sweeps; ++s) {
      ICS_LAUNCH(h, ICS_K_JACOBI,
                 k_jacobi_sweep<TB, TV><<<grid_for(N, 128), 128, 0, st>>>(h.m, (const TB*)h.blk, (const TB*)h.dginv,
                                                                          h.src, x, y));
      TV* tmp = x;
      x = y;
      y = tmp;
    }
    spmv_t<TB, TV>(h, x, t);
    ICS_LAUNCH(h, ICS_K_VECTOR,
               k_resid<TV><<<inst_grid(h), RB, 0, st>>>(h.m.Nc, h.src, t, r, h.partials, h.counter, ks->res));
    ICS_CUDA(cudaGetLastError());
    ICS_CUDA(cudaMemcpyAsync(h.ksHost->res, ks->res, 5 * h.m.nInst * sizeof(double), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaStreamSynchronize(st));
    finite = final_residuals(h, nf, p);
    p.nIter += h.cfg.c.n_sweeps;
    if (!finite) break;
  } while (!stop_test(h, p));
  ICS_LAUNCH(h, ICS_K_VECTOR,
             k_to_dW<TV><<<grid_for(N, 256), 256, 0, st>>>(N, x, h.dW, h.m.solD[0], h.m.solD[1], h.m.solD[2]));
  ICS_CUDA(cudaGetLastError());
  return finite ? ICS_OK : ICS_ERR_NONFINITE;
}


// the error of a solve from its status flags
static int krylov_error(int status) {
  return status & 8 ? ICS_ERR_TIMEOUT : status & 4 ? ICS_ERR_NONFINITE : ICS_ERR_BREAKDOWN;
}

template <typename TB, typename TV>
static int gmres_t(Handle& h, ResIO& p) {
  const int N = h.m.N, m = h.cfg.c.n_directions;
  const long n5 = 5L * N;
  const long vs = (long)kstride(h);
  cudaStream_t st = h.stream;
  KrylovScalars* ks = h.ks;
  TV* V = (TV*)h.kv;
  TV* w = (TV*)h.kw;
  TV* x = (TV*)h.kx;
  TV* t = (TV*)h.kt;
  std::vector<double> nf;
  norm_factors_t<TB, TV>(h, nf, p);
  column_reset(h, m);
  // r = b, x = 0
  ICS_CUDA(cudaMemsetAsync(x, 0, n5 * sizeof(TV), st));
  to_vec(h, h.src, w);
  int status = ICS_OK;
  // one restart cycle: every scalar it needs lives in device memory, so the
  // same launch sequence can be captured once and replayed per cycle
  auto cycle = [&]() {
    precondition_t<TB, TV>(h, w);
    krylov_column(h, sizeof(TV) == 4, n5, w, V, vs, -1, m);
    for (int i = 0; i < m; ++i) {
      const TV* vi = V + (size_t)i * vs;
      if (!fused_op_t<TB, TV>(h, vi, w)) {
        spmv_t<TB, TV>(h, vi, w);
        precondition_t<TB, TV>(h, w);
      }
      krylov_column(h, sizeof(TV) == 4, n5, w, V, vs, i, m);
    }
    ICS_LAUNCH(h, ICS_K_SCALAR, k_backsub<<<1, 32, 0, st>>>(ks, m));
    ICS_LAUNCH(h, ICS_K_VECTOR, k_xupdate<TV><<<pass_grid(n5 / V16<TV>::n), RB, 0, st>>>(n5, x, V, ks, m, vs));
    spmv_t<TB, TV>(h, x, t);
    ICS_LAUNCH(h, ICS_K_VECTOR,
               k_resid<TV><<<inst_grid(h), RB, 0, st>>>(h.m.Nc, h.src, t, w, h.partials, h.counter, ks->res));
  };
  // the captured launches hold DevMesh by value: the non-LF viscous block
  // parts (m.vjslot) are part of the key
  const int key = (h.m.vjslot ? 10000000 : 0) + h.cfg.c.preconditioner * 100000 + prec(h) * 1000 + m;
  const bool useGraph = !h.prof;  // per-launch event timing needs direct launches
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
    h.launches = before;  // captured, not executed
    h.cycleKey = key;
  }
  do {
    if (useGraph) {
      ICS_CUDA(cudaGraphLaunch(h.cycleExec, st));
      h.launches += h.cycleLaunches;
    } else {
      cycle();
    }
    ICS_CUDA(cudaGetLastError());
    ICS_CUDA(cudaMemcpyAsync(h.ksHost->res, ks->res, 5 * h.m.nInst * sizeof(double), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaMemcpyAsync(&h.ksHost->status, &ks->status, sizeof(int), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaStreamSynchronize(st));
    if (h.ksHost->status) {
      status = krylov_error(h.ksHost->status);
      p.nIter++;
      break;
    }
    const bool finite = final_residuals(h, nf, p);
    p.nIter++;
    if (!finite) {
      status = ICS_ERR_NONFINITE;
      break;
    }
  } while (!stop_test(h, p));
  ICS_LAUNCH(h, ICS_K_VECTOR, k_to_dW<TV><<<grid_for(N, 256), 256, 0, st>>>(N, x, h.dW, h.m.solD[0], h.m.solD[1], h.m.solD[2]));
  ICS_CUDA(cudaGetLastError());
  return status;
}

int gmres_solve(Handle& h, ics_solver_perf* perf, std::vector<double>& initRes) {
  ResIO r;
  int st;
  if (h.cfg.c.solver == ICS_SOLVER_SMOOTH)
    st = prec(h) == ICS_PREC_MIXED ? smooth_t<float, float>(h, r) : smooth_t<double, double>(h, r);
  else
    st = prec(h) == ICS_PREC_MIXED ? gmres_t<float, float>(h, r) : gmres_t<double, double>(h, r);
  // the C ABI's summary: maximum over instances per equation
  memset(perf, 0, sizeof(*perf));
  for (int k = 0; k < 5; ++k) {
    perf->init_res[k] = -VGREAT;
    perf->final_res[k] = -VGREAT;
    for (int J = 0; J < h.m.nInst; ++J) {
      perf->init_res[k] = fmax(perf->init_res[k], r.init[5 * J + k]);
      perf->final_res[k] = fmax(perf->final_res[k], r.fin[5 * J + k]);
    }
  }
  perf->n_iterations = r.nIter;
  perf->converged = st == ICS_OK;
  initRes = r.init;
  return st;
}

// ------------------------------------------------------------ autotuner
// Times the Krylov-side launch choices on the handle's assembled system with
// CUDA events on its stream (median of three runs each, after a warm-up):
// the fused LU-SGS operator against SpMV plus separate sweeps, and the rows
// per thread of the reverse sweep.  Sets the fastest; the arithmetic of every choice is the
// same up to the order of the sums.
template <typename TB, typename TV>
static void autotune_linalg_t(Handle& h, std::vector<std::pair<std::string, double>>& log) {
  cudaStream_t st = h.stream;
  TV* V = (TV*)h.kv;
  TV* w = (TV*)h.kw;
  TV* t = (TV*)h.kt;
  cudaEvent_t e0, e1;
  ICS_CUDA(cudaEventCreate(&e0));
  ICS_CUDA(cudaEventCreate(&e1));
  auto timed = [&](auto&& fn) {
    fn();
    double best[5];
    for (int r = 0; r < 5; ++r) {
      ICS_CUDA(cudaEventRecord(e0, st));
      fn();
      ICS_CUDA(cudaEventRecord(e1, st));
      ICS_CUDA(cudaEventSynchronize(e1));
      float ms = 0;
      ICS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      best[r] = ms;
    }
    std::sort(best, best + 5);
    return best[2];
  };
  // operand: v_0 = b
  to_vec(h, h.src, V);
  ICS_CUDA(cudaMemsetAsync(&h.ks->status, 0, sizeof(int), st));
  h.tuneFused = 1;
  if (fused_op_available<TB, TV>(h)) {
    const double fused = timed([&]() { fused_op_t<TB, TV>(h, V, w); });
    const double split = timed([&]() {
      spmv_t<TB, TV>(h, V, t);
      precondition_t<TB, TV>(h, t);
    });
    log.emplace_back("operator_fused", fused);
    log.emplace_back("operator_spmv_then_lusgs", split);
    h.tuneFused = fused <= split ? 1 : 0;
  }
  // rows per thread of the reverse level sweeps, timed on the whole LU-SGS,
  // where a level takes the kernels they choose between
  h.tuneRevRows = 1;
  if (!rev_rows_choice<TB>(h)) {
    ICS_CUDA(cudaEventDestroy(e0));
    ICS_CUDA(cudaEventDestroy(e1));
    ICS_CUDA(cudaGetLastError());
    return;
  }
  double revMs[3] = {0, 0, 0};
  for (int rows : {1, 2}) {
    h.tuneRevRows = rows;
    revMs[rows] = timed([&]() {
      to_vec(h, h.src, t);
      precondition_t<TB, TV>(h, t);
    });
    log.emplace_back("reverse_rows_" + std::to_string(rows), revMs[rows]);
  }
  h.tuneRevRows = revMs[2] < revMs[1] ? 2 : 1;
  ICS_CUDA(cudaEventDestroy(e0));
  ICS_CUDA(cudaEventDestroy(e1));
  ICS_CUDA(cudaGetLastError());
}

void autotune_linalg(Handle& h, std::vector<std::pair<std::string, double>>& log) {
  if (prec(h) == ICS_PREC_MIXED)
    autotune_linalg_t<float, float>(h, log);
  else
    autotune_linalg_t<double, double>(h, log);
}

// sum of a device array (deterministic fixed-order reduction)
double device_sum(Handle& h, const double* a, int n) {
  ICS_LAUNCH(h, ICS_K_VECTOR, k_sumsq<<<reduce_grid(n), RB, 0, h.stream>>>(n, a, h.partials, h.counter, &h.ks->red[8]));
  double v = 0;
  ICS_CUDA(cudaMemcpyAsync(&v, &h.ks->red[8], sizeof(double), cudaMemcpyDeviceToHost, h.stream));
  ICS_CUDA(cudaStreamSynchronize(h.stream));
  return v;
}

// rho L2 residual: sqrt(sum (div(phi) V)^2) from the per-cell squares, and
// whether every entry of the source is finite; host_src (if not null) receives
// the source in the same wait
double rho_l2(Handle& h, double* host_src, bool* finite) {
  ICS_LAUNCH(h, ICS_K_VECTOR, k_sumsq<<<reduce_grid(h.m.N), RB, 0, h.stream>>>(h.m.N, h.scratch, h.partials, h.counter, &h.ks->l2));
  struct {
    double l2;
    int nonfinite, status;
  } v = {0, 0, 0};
  static_assert(offsetof(KrylovScalars, nonfinite) == offsetof(KrylovScalars, l2) + sizeof(double), "");
  ICS_CUDA(cudaMemcpyAsync(&v, &h.ks->l2, sizeof(v), cudaMemcpyDeviceToHost, h.stream));
  if (host_src)
    ICS_CUDA(cudaMemcpyAsync(host_src, h.src, 5ull * h.m.N * sizeof(double), cudaMemcpyDeviceToHost, h.stream));
  ICS_CUDA(cudaStreamSynchronize(h.stream));
  *finite = v.nonfinite == 0;
  return std::sqrt(v.l2);
}

// ------------------------------------------------------ passive scalar
// The 1x0 coupled system of the scalar transport (same GMRES, LU-SGS and
// norm factors as the flow's, one equation): 1x1 sliced-ELL blocks, FP64.
__global__ void __launch_bounds__(128) k_s_spmv(DevMesh m, const double* __restrict__ blk,
                                                const double* __restrict__ dg, const double* __restrict__ x,
                                                double* __restrict__ y) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.N) return;
  const int s = c >> 5, lane = c & 31;
  double acc = dg[c] * x[c];
  const int base = m.slot_base[s];
  for (int t = 0; t < m.nslot[c]; ++t) {
    const int col = m.scol[(base + t) * 32 + lane];
    acc += blk[(size_t)(base + t) * 32 + lane] * x[col];
  }
  y[c] = acc;
}

__device__ __forceinline__ void s_fwd_row(const DevMesh& m, const double* __restrict__ blk,
                                          const double* __restrict__ rD, double* __restrict__ r, int c, bool scale) {
  const int s = c >> 5, lane = c & 31;
  const int base = m.slot_base[s];
  double acc = r[c];
  for (int t = 0; t < m.nlow[c]; ++t) {
    const int col = m.scol[(base + t) * 32 + lane];
    acc -= blk[(size_t)(base + t) * 32 + lane] * (rD[col] * r[col]);
  }
  r[c] = scale ? rD[c] * acc : acc;
}

__device__ __forceinline__ void s_rev_row(const DevMesh& m, const double* __restrict__ blk,
                                          const double* __restrict__ rD, double* __restrict__ r, int c) {
  const int s = c >> 5, lane = c & 31;
  const int base = m.slot_base[s];
  double acc = r[c];
  for (int t = m.nslot[c] - 1; t >= m.nlow[c]; --t) {
    const int col = m.scol[(base + t) * 32 + lane];
    acc -= blk[(size_t)(base + t) * 32 + lane] * r[col];
  }
  r[c] = rD[c] * acc;
}

template <int MODE>
__global__ void __launch_bounds__(128) k_s_lusgs_level(DevMesh m, const double* __restrict__ blk,
                                                       const double* __restrict__ rD, double* __restrict__ r,
                                                       const int* __restrict__ cells, int start, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int c = cells ? cells[start + i] : start + i;
  if (MODE == 1)
    s_rev_row(m, blk, rD, r, c);
  else
    s_fwd_row(m, blk, rD, r, c, MODE == 2);
}

template <bool FWD>
__global__ void __launch_bounds__(1024) k_s_lusgs_block(DevMesh m, const double* __restrict__ blk,
                                                        const double* __restrict__ rD, double* __restrict__ r,
                                                        const int* __restrict__ cells, const int* __restrict__ lptr,
                                                        int nlev) {
  for (int l = 0; l < nlev; ++l) {
    for (int i = lptr[l] + threadIdx.x; i < lptr[l + 1]; i += blockDim.x) {
      if (FWD)
        s_fwd_row(m, blk, rD, r, cells[i], false);
      else
        s_rev_row(m, blk, rD, r, cells[i]);
    }
    __syncthreads();
  }
}

__global__ void k_s_jacobi(int N, const double* __restrict__ dg, double* __restrict__ r) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < N) r[c] /= dg[c];
}

// out[0] = sum w
__global__ void __launch_bounds__(RB) k_s_sum(int N, const double* __restrict__ w, double* __restrict__ partials,
                                              unsigned int* __restrict__ counter, double* __restrict__ out) {
  double acc[1] = {0.0};
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) acc[0] += w[c];
  reduce_finish<1>(acc, partials, counter, out);
}

__global__ void k_s_wmavg(int N, const double* __restrict__ w, const double* __restrict__ sum,
                          double* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < N) out[c] = w[c] - sum[0] / N;
}

// out[0] = sum |t| + |b|, out[1] = sum |b|
__global__ void __launch_bounds__(RB) k_s_normfac(int N, const double* __restrict__ b, const double* __restrict__ t,
                                                  double* __restrict__ partials, unsigned int* __restrict__ counter,
                                                  double* __restrict__ out) {
  double acc[2] = {0.0, 0.0};
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
    acc[0] += fabs(t[c]) + fabs(b[c]);
    acc[1] += fabs(b[c]);
  }
  reduce_finish<2>(acc, partials, counter, out);
}

// r = b - t, out[0] = sum |r|
__global__ void __launch_bounds__(RB) k_s_resid(int N, const double* __restrict__ b, const double* __restrict__ t,
                                                double* __restrict__ r, double* __restrict__ partials,
                                                unsigned int* __restrict__ counter, double* __restrict__ out) {
  double acc[1] = {0.0};
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
    const double v = b[c] - t[c];
    r[c] = v;
    acc[0] += fabs(v);
  }
  reduce_finish<1>(acc, partials, counter, out);
}

// scalar cyclic interfaces: y_c += sum over c's cyclic faces of a_f x_partner
// (a_f in the upper slot of the scalar face coefficients)
__global__ void k_s_cyc_mv(DevMesh m, const double* __restrict__ sface, int FB, const double* __restrict__ x,
                           double* __restrict__ y) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= m.ncrow) return;
  const int c = m.cyc_row[r];
  double acc = y[c];
  for (int e = m.cyc_ptr[r]; e < m.cyc_ptr[r + 1]; ++e) {
    const int b = m.cyc_face[e];
    acc += sface[FB + m.F + b] * x[m.bpartner[b]];
  }
  y[c] = acc;
}

static void s_spmv(Handle& h, const double* x, double* y) {
  ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_spmv<<<grid_for(h.m.N, 128), 128, 0, h.stream>>>(h.m, h.sblk, h.sdg, x, y));
  if (h.m.ncrow)
    ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_cyc_mv<<<grid_for(h.m.ncrow, 128), 128, 0, h.stream>>>(h.m, h.sface, h.m.F + h.m.B,
                                                                                            x, y));
}

static void s_precondition(Handle& h, double* r) {
  const DevMesh& m = h.m;
  const int pc = h.cfg.c.preconditioner;
  if (pc == ICS_PC_JACOBI) {
    ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_jacobi<<<grid_for(m.N, 256), 256, 0, h.stream>>>(m.N, h.sdg, r));
    return;
  }
  if (pc != ICS_PC_LUSGS) return;
  if ((long)m.N < 2048L * m.nfl) {
    ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_lusgs_block<true><<<1, 1024, 0, h.stream>>>(m, h.sblk, h.srD, r, m.fl_cells,
                                                                                  m.fl_lptr, m.nfl));
  } else {
    for (int l = 1; l < m.nfl; ++l) {  // level 0 has no lower neighbours
      const int a = m.fl_ptr[l], cnt = m.fl_ptr[l + 1] - a;
      const bool contig = m.fl_cstart[l] >= 0;
      ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_lusgs_level<0><<<grid_for(cnt, 128), 128, 0, h.stream>>>(
                                       m, h.sblk, h.srD, r, contig ? nullptr : m.fl_cells,
                                       contig ? m.fl_cstart[l] : a, cnt));
    }
  }
  if ((long)m.N < 2048L * m.nrl) {
    ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_lusgs_block<false><<<1, 1024, 0, h.stream>>>(m, h.sblk, h.srD, r, m.rl_cells,
                                                                                   m.rl_lptr, m.nrl));
  } else {
    for (int l = 0; l < m.nrl; ++l) {
      const int a = m.rl_ptr[l], cnt = m.rl_ptr[l + 1] - a;
      const bool contig = m.rl_cstart[l] >= 0;
      ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_lusgs_level<1><<<grid_for(cnt, 128), 128, 0, h.stream>>>(
                                       m, h.sblk, h.srD, r, contig ? nullptr : m.rl_cells,
                                       contig ? m.rl_cstart[l] : a, cnt));
    }
  }
}

// gmres::solveDelta on the scalar system: b = h.ssrc, norm factors from the
// previous-iteration rhoS, increment in dx
int scalar_gmres(Handle& h, double* dx, ics_solver_perf* perf) {
  const int N = h.m.N, m = h.cfg.c.n_directions;
  cudaStream_t st = h.stream;
  KrylovScalars* ks = h.ks;
  const long vs = ((long)N + 63) / 64 * 64;
  double* V = (double*)h.kv;
  double* w = (double*)h.kw;
  double* t = (double*)h.kt;
  double* red = ks->red;
  ICS_CUDA(cudaMemsetAsync(&ks->status, 0, sizeof(int), st));
  ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_sum<<<reduce_grid(N), RB, 0, st>>>(N, h.srhoS, h.partials, h.counter, &red[2]));
  ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_wmavg<<<grid_for(N, 256), 256, 0, st>>>(N, h.srhoS, &red[2], w));
  s_spmv(h, w, t);
  ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_normfac<<<reduce_grid(N), RB, 0, st>>>(N, h.ssrc, t, h.partials, h.counter, &red[3]));
  double hv[2];
  ICS_CUDA(cudaMemcpyAsync(hv, &red[3], 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
  ICS_CUDA(cudaStreamSynchronize(st));
  const double nf = hv[0] + VSMALL;
  memset(perf, 0, sizeof(*perf));
  perf->init_res[0] = perf->final_res[0] = hv[1] / nf;
  column_reset(h, m);
  ICS_CUDA(cudaMemsetAsync(dx, 0, N * sizeof(double), st));
  ICS_CUDA(cudaMemcpyAsync(w, h.ssrc, N * sizeof(double), cudaMemcpyDeviceToDevice, st));
  const ics_config& cf = h.cfg.c;
  int status = ICS_OK;
  while (true) {
    s_precondition(h, w);
    krylov_column(h, false, N, w, V, vs, -1, m);
    for (int i = 0; i < m; ++i) {
      s_spmv(h, V + (size_t)i * vs, w);
      s_precondition(h, w);
      krylov_column(h, false, N, w, V, vs, i, m);
    }
    ICS_LAUNCH(h, ICS_K_SCALAR, k_backsub<<<1, 32, 0, st>>>(ks, m));
    ICS_LAUNCH(h, ICS_K_VECTOR, k_xupdate<double><<<pass_grid(N / 2), RB, 0, st>>>(N, dx, V, ks, m, vs));
    s_spmv(h, dx, t);
    ICS_LAUNCH(h, ICS_K_PASSIVE, k_s_resid<<<reduce_grid(N), RB, 0, st>>>(N, h.ssrc, t, w, h.partials, h.counter,
                                                                         &red[5]));
    double rs = 0;
    int stt = 0;
    ICS_CUDA(cudaMemcpyAsync(&rs, &red[5], sizeof(double), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaMemcpyAsync(&stt, &ks->status, sizeof(int), cudaMemcpyDeviceToHost, st));
    ICS_CUDA(cudaStreamSynchronize(st));
    perf->n_iterations++;
    if (stt) {
      status = krylov_error(stt);
      break;
    }
    perf->final_res[0] = rs / nf;
    if (!std::isfinite(perf->final_res[0])) {
      status = ICS_ERR_NONFINITE;
      break;
    }
    if (perf->n_iterations < cf.min_iter) continue;
    const double rel = perf->final_res[0] / (perf->init_res[0] + ROOTVSMALL);
    if (perf->n_iterations >= cf.max_iter || perf->final_res[0] < cf.tolerance || rel < cf.rel_tol) break;
  }
  perf->converged = status == ICS_OK;
  ICS_CUDA(cudaGetLastError());
  return status;
}

}  // namespace ics
