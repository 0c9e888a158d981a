// LU-SGS sweeps of a chain: a mesh whose rows couple to the row before and the
// row after only (a one-dimensional mesh in its natural numbering).
//
// Both sweeps of lusgs.C:220-385 are then first-order recurrences along the
// chain with 5x5 coefficients that do not change while the matrix stands:
//   forward  r'_c = r_c - L_c (rD_{c-1} r'_{c-1})
//   reverse  z_c  = rD_c (r'_c - U_c z_{c+1})
// i.e. x_p = b_p + M_p x_{p-1} over positions p (p = c forward, N-1-c
// reverse).  Swept row after row that is N dependent steps of an L2 round trip
// each (1.5 us); as a scan it is a few dozen.  The positions are cut into
// CHAIN_CHUNKS chunks of equal length; per matrix, k_chain_products and
// k_chain_tables compute the products of the M (of a chunk, of runs of chunks,
// of runs of blocks), and one cluster of 8 blocks applies both sweeps:
//   1. every chunk's recurrence from a zero inflow (8 lanes per chunk, one
//      component each),
//   2. the chunks' ends by a scan over the block's 16 chunks (4 steps), then
//      the blocks' ends, gathered through distributed shared memory,
//   3. every chunk's recurrence again, from the inflow found in 2.
// The rows come from step 3, in the arithmetic of the row-by-row sweep, so the
// products' rounding reaches them only through a chunk's inflow.  Everything
// is FP64 in both precisions (the mixed path rounds once, to its FP32
// result).  Bound by dependent FP64 instructions (64 cycles each):
// 20 us for both sweeps of 1000 rows, 1.8 ms by the sync-free sweeps.
#include <cooperative_groups.h>

#include "blocks.cuh"
#include "ics_internal.cuh"

namespace ics {

namespace {

namespace cg = cooperative_groups;

constexpr int CHAIN_BLOCKS = 8;                             // blocks of the cluster
constexpr int BLOCK_CHUNKS = 16;                            // chunks per block
constexpr int CHAIN_CHUNKS = CHAIN_BLOCKS * BLOCK_CHUNKS;   // chunks of the chain
constexpr int SCAN_STEPS = 4;                               // log2(BLOCK_CHUNKS)

// Tables of one sweep direction (5x5 matrices, row-major).  Per position: B,
// the block that couples it to the position before, and d, the rD of the
// position before (forward) or its own (reverse).  Per chunk k: T[s], the
// product of the M of the 2^s chunks ending at k, and G, of its block's chunks
// up to k.  Q[j][i]: of the blocks i+1 .. j-1.
struct ChainTab {
  double *B, *d, *T, *G, *Q;
};

__host__ __device__ inline size_t chain_words(size_t N) {
  return 26 * N + 25 * ((SCAN_STEPS + 1) * CHAIN_CHUNKS + CHAIN_BLOCKS * CHAIN_BLOCKS);
}

__host__ __device__ inline ChainTab chain_tab(double* base, size_t N, int dir) {
  ChainTab t;
  t.B = base + dir * chain_words(N);
  t.d = t.B + 25 * N;
  t.T = t.d + N;
  t.G = t.T + 25 * SCAN_STEPS * CHAIN_CHUNKS;
  t.Q = t.G + 25 * CHAIN_CHUNKS;
  return t;
}

// C = A B of 5x5 matrices spread over lanes 5 i + j of a warp
__device__ __forceinline__ double warp_mul(double a, double b, int i, int j) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 5; ++k)
    s += __shfl_sync(0xffffffffu, a, 5 * i + k) * __shfl_sync(0xffffffffu, b, 5 * k + j);
  return s;
}

// one warp per (direction, chunk): B, d and the chunk's product T[0]
template <typename TB>
__global__ void __launch_bounds__(32) k_chain_products(DevMesh m, const TB* __restrict__ blk,
                                                       const TB* __restrict__ rD, double* base, int len) {
  const int dir = blockIdx.x / CHAIN_CHUNKS, k = blockIdx.x % CHAIN_CHUNKS;
  const int N = m.N;
  const ChainTab t = chain_tab(base, N, dir);
  const bool on = threadIdx.x < 25;
  const int lane = on ? threadIdx.x : 0;
  const int i = lane / 5, j = lane % 5;
  double P = 0.0;  // stays 0 for a chunk past the end of a short chain
  const long p0 = (long)k * len, p1 = p0 + len < N ? p0 + len : N;
  for (long p = p0; p < p1; ++p) {
    const int c = dir ? N - 1 - (int)p : (int)p;
    const int s = c >> 5, cl = c & 31;
    const int nl = m.nlow[c];
    double e = 0.0, d = dir ? double(rD[c]) : 0.0;
    if (p > 0) {  // the chain is unbroken: every position but the first has the one before
      const size_t slot = m.slot_base[s] + (dir ? nl : 0);
      if constexpr (sizeof(TB) == 8) {
        e = blk[(slot * 25 + lane) * 32 + cl];
      } else {
        SlotBlock<TB> Bk;
        Bk.load(blk, slot, cl);
        e = Bk.entry(m.gamma, i, j);
      }
      if (m.vjslot) e -= vj_entry<TB>(m, slot, cl, dir ? c + 1 : c - 1, i, j);
      if (!dir) d = double(rD[c - 1]);
    }
    const double M = -d * e;
    const double prod = warp_mul(M, P, i, j);
    P = p == p0 ? M : prod;
    if (on) t.B[25 * p + lane] = e;
    if (threadIdx.x == 0) t.d[p] = d;
  }
  if (on) t.T[25 * k + lane] = P;
}

// one block of 16 warps per direction: the products of chunks and blocks
__global__ void __launch_bounds__(512) k_chain_tables(int N, double* base) {
  const ChainTab t = chain_tab(base, N, blockIdx.x);
  const int warp = threadIdx.x >> 5, lane = (threadIdx.x & 31) < 25 ? (threadIdx.x & 31) : 0;
  const bool on = (threadIdx.x & 31) < 25;
  const int i = lane / 5, j = lane % 5;
  double* T = t.T;
  for (int s = 1; s < SCAN_STEPS; ++s) {
    const int half = 1 << (s - 1);
    const double* A = T + 25 * (s - 1) * CHAIN_CHUNKS;
    for (int k = warp; k < CHAIN_CHUNKS; k += 16) {
      if (k % BLOCK_CHUNKS < half) continue;
      const double v = warp_mul(A[25 * k + lane], A[25 * (k - half) + lane], i, j);
      if (on) T[25 * (s * CHAIN_CHUNKS + k) + lane] = v;
    }
    __syncthreads();
  }
  if (warp < CHAIN_BLOCKS) {
    double g = 0.0;
    for (int q = 0; q < BLOCK_CHUNKS; ++q) {
      const int k = warp * BLOCK_CHUNKS + q;
      const double e = T[25 * k + lane], v = warp_mul(e, g, i, j);
      g = q == 0 ? e : v;
      if (on) t.G[25 * k + lane] = g;
    }
  }
  __syncthreads();
  if (warp < CHAIN_BLOCKS) {
    double q = i == j ? 1.0 : 0.0;
    for (int b = warp - 1; b >= 0; --b) {
      if (on) t.Q[25 * (warp * CHAIN_BLOCKS + b) + lane] = q;
      q = warp_mul(q, t.G[25 * (b * BLOCK_CHUNKS + BLOCK_CHUNKS - 1) + lane], i, j);
    }
  }
}

// A chunk's recurrence over positions p0 .. p1-1 with inflow xj (component j
// of the position before p0; this lane's component is i), the next position's
// coefficients in flight; write(c, x) takes every row.  Returns the last x.
template <int DIR, typename In, typename Write>
__device__ __forceinline__ double chain_chunk(int N, const ChainTab& t, long p0, long p1, int i, unsigned mask,
                                              double x, In in, Write write) {
  auto cell = [&](long p) { return DIR ? N - 1 - (int)p : (int)p; };
  double b = 0.0, d = 0.0, B[5] = {0, 0, 0, 0, 0};
  auto load = [&](long p) {
    b = in(cell(p));
    d = t.d[p];
#pragma unroll
    for (int j = 0; j < 5; ++j) B[j] = t.B[25 * p + 5 * i + j];
  };
  if (p0 < p1) load(p0);
  for (long p = p0; p < p1; ++p) {
    const double bp = b, dp = d, Bp[5] = {B[0], B[1], B[2], B[3], B[4]};
    if (p + 1 < p1) load(p + 1);
    const double u = DIR ? x : dp * x;
    double y = 0.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) y += Bp[j] * __shfl_sync(mask, u, j, 8);
    x = DIR ? dp * (bp - y) : bp - y;
    write(cell(p), x);
  }
  return x;
}

// One sweep.  in(c): component i of row c's right-hand side; out(c, x) takes
// the result.
template <int DIR, typename In, typename Write>
__device__ __forceinline__ void chain_sweep(int N, int len, const ChainTab& t, In in, Write out,
                                            double (*v)[BLOCK_CHUNKS][5], double (*part)[5]) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int grp = threadIdx.x >> 3, i8 = threadIdx.x & 7, i = i8 < 5 ? i8 : 0;
  const bool on = i8 < 5;
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  const int k = rank * BLOCK_CHUNKS + grp;
  const long p0 = (long)k * len, p1 = p0 + len < N ? p0 + len : N;
  auto inRow = [&](int c) { return in(c, i); };
  const double x = chain_chunk<DIR>(N, t, p0, p1, i, mask, 0.0, inRow, [](int, double) {});
  if (on) v[0][grp][i] = x;
  __syncthreads();
  // the ends of the block's chunks
  int cur = 0;
#pragma unroll
  for (int s = 0; s < SCAN_STEPS; ++s) {
    const int back = 1 << s;
    double a = v[cur][grp][i];
    if (grp >= back) {
      const double* T = t.T + 25 * ((size_t)s * CHAIN_CHUNKS + k) + 5 * i;
#pragma unroll
      for (int j = 0; j < 5; ++j) a += T[j] * v[cur][grp - back][j];
    }
    if (on) v[cur ^ 1][grp][i] = a;
    cur ^= 1;
    __syncthreads();
  }
  // the inflow of this block: the ends of the blocks before it
  cluster.sync();
  if (grp < CHAIN_BLOCKS && on) {
    double a = 0.0;
    if (grp < rank) {
      const double* end = cluster.map_shared_rank(&v[cur][BLOCK_CHUNKS - 1][0], grp);
      const double* Q = t.Q + 25 * (rank * CHAIN_BLOCKS + grp) + 5 * i;
#pragma unroll
      for (int j = 0; j < 5; ++j) a += Q[j] * end[j];
    }
    part[grp][i] = a;
  }
  __syncthreads();
  double xin = 0.0;
  for (int g = 0; g < rank; ++g) xin += part[g][i];
  if (grp > 0) {
    const double* G = t.G + 25 * (size_t)(k - 1) + 5 * i;
    double a = v[cur][grp - 1][i];
#pragma unroll
    for (int j = 0; j < 5; ++j) a += G[j] * __shfl_sync(mask, xin, j, 8);
    xin = a;
  }
  chain_chunk<DIR>(N, t, p0, p1, i, mask, xin, inRow, [&](int c, double r) {
    if (on) out(c, i, r);
  });
}

template <typename TV>
__global__ void __cluster_dims__(CHAIN_BLOCKS, 1, 1) __launch_bounds__(8 * BLOCK_CHUNKS)
    k_chain_sweeps(int N, int len, double* base, TV* r, double* fwd) {
  __shared__ double v[2][BLOCK_CHUNKS][5];
  __shared__ double part[CHAIN_BLOCKS][5];
  chain_sweep<0>(
      N, len, chain_tab(base, N, 0), [&](int c, int i) { return double(r[5 * (size_t)c + i]); },
      [&](int c, int i, double x) { fwd[5 * (size_t)c + i] = x; }, v, part);
  __threadfence();
  cg::this_cluster().sync();  // other blocks read these rows of fwd; v is reused
  chain_sweep<1>(
      N, len, chain_tab(base, N, 1), [&](int c, int i) { return __ldcg(fwd + 5 * (size_t)c + i); },
      [&](int c, int i, double x) { r[5 * (size_t)c + i] = TV(x); }, v, part);
  cg::this_cluster().sync();  // the other blocks have read v
}

int chain_len(int N) { return (N + CHAIN_CHUNKS - 1) / CHAIN_CHUNKS; }

template <typename TB>
void setup_t(Handle& h) {
  const int N = h.m.N;
  ICS_LAUNCH(h, ICS_K_JAC_ROWS,
             k_chain_products<TB><<<2 * CHAIN_CHUNKS, 32, 0, h.stream>>>(h.m, (const TB*)h.blk, (const TB*)h.rD,
                                                                         h.m.chain, chain_len(N)));
  ICS_LAUNCH(h, ICS_K_JAC_ROWS, k_chain_tables<<<2, 512, 0, h.stream>>>(N, h.m.chain));
}

template <typename TV>
void sweeps_t(Handle& h, TV* r) {
  const int N = h.m.N;
  ICS_LAUNCH(h, ICS_K_LUSGS_FWD,
             k_chain_sweeps<TV><<<CHAIN_BLOCKS, 8 * BLOCK_CHUNKS, 0, h.stream>>>(N, chain_len(N), h.m.chain, r,
                                                                                 (double*)h.m.sweep_pad));
}

}  // namespace

size_t chain_table_words(int N) { return 2 * chain_words(N); }

void chain_setup(Handle& h) {
  if (prec(h) == ICS_PREC_MIXED)
    setup_t<float>(h);
  else
    setup_t<double>(h);
  ICS_CUDA(cudaGetLastError());
}

void chain_sweeps(Handle& h, void* r) {
  if (prec(h) == ICS_PREC_MIXED)
    sweeps_t<float>(h, (float*)r);
  else
    sweeps_t<double>(h, (double*)r);
  ICS_CUDA(cudaGetLastError());
}

}  // namespace ics
