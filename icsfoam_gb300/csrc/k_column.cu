// One column of the Arnoldi process in one launch: the modified Gram-Schmidt
// of a new Krylov vector against the basis (gmres.C:936-1011) and its
// normalisation.
//
//   for j = 0 .. dir:  h_j = w . v_j;  w -= h_j v_j
//   beta = |w|;  v_{dir+1} = w / beta
//
// (dir = -1, the start of a cycle, has the last line only.)  Every step needs
// the sum of the step before over the whole vector.  As one launch per step
// that was dir + 2 launches, each reading w and two basis vectors and writing
// w back, with a reduction tail of its own: 13 us per step at 1M cells in
// FP32 (84 MB, partly from L2), 4-5 us on small meshes.  Here a cooperative
// grid of one block per SM keeps its slice of w in registers for the whole
// column, streams each basis vector once through shared memory -- with the
// next one's copies in flight while the sum is exchanged -- and the blocks
// exchange their partial sums through one slot each: a block polls all slots
// of the step and adds them up itself, in slot order, so every block has the
// same h_j after one L2 round trip and the sums are reproducible.
//
// The slots start as a sentinel (all bits set, which no sum is published as)
// and are written once per column; a column resets the slots of the next one.
// The waits are bounded: a block whose wait runs out sets status bit 8, and from
// then on every wait of every block ends within 64 polls, with a NaN for a sum
// (the solve reports the flag; a test of it in each step would cost 1% of a
// small system's solve).  One further block, outside the exchange, rotates the
// Hessenberg column of the direction before.
//
// FP32 sums: a thread adds runs of RUN chunks (4 to 12 products, no more than
// one launch per step gave a thread at that size) and of 32 products of what
// its registers do not hold in FP32; the runs are joined with their rounding
// errors kept, and everything across threads is FP64.  Error of w . v of
// random vectors against 64 bits, of |w| |v|: 1M cells 1.9e-11 (one launch per
// step 2.2e-11, two runs of up to 36 products here 3.2e-11), 117k cells 5.8e-11
// (5.8e-11, 7.1e-11).
//
// Measured, the columns of a cycle of 8 directions (45 steps, 9 launches; one
// launch per step before: 540 us at 1M cells in FP32): 323 us at 1M cells in
// FP32, where the exchange (2.3 of 6.6 us a step) and the half vector that does
// not fit beside the rest on chip bound it; 349 us at 197k cells in FP64, bound
// by the FP64 pipe; 117 us at 10k cells, the exchange and the block sums (about
// 1 us each).
#include <algorithm>
#include <type_traits>

#include "krylov.cuh"

namespace ics {

namespace {

constexpr int COLUMN_SPIN_LIMIT = 1 << 20;
constexpr int MAX_GRID = 160;  // blocks of the exchange at most (five slots per polling lane)
// Blocks of the exchange, and the pauses (ns) of a polling warp before its
// first and between its polls.  All blocks poll the lines that all blocks have
// still to write, and polls that come too early hold those stores up: without
// the pauses an exchange of 151 blocks takes 3900 cycles instead of 2300, one
// of 128 blocks 2600 instead of 1800; few blocks do best without.
constexpr int SMALL_GRID = 128;
constexpr int PAUSE_BLOCKS = 32, PAUSE_FIRST = 300, PAUSE_NEXT = 60;

__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

__device__ __forceinline__ void zero16(float4& x) { x = make_float4(0, 0, 0, 0); }
__device__ __forceinline__ void zero16(double2& x) { x = make_double2(0, 0); }

// elements at and past n of 16-byte chunk q read as zero
template <typename TV>
__device__ __forceinline__ typename V16<TV>::T load16(const TV* p, long q, long n) {
  using VT = typename V16<TV>::T;
  constexpr int L = V16<TV>::n;
  VT v;
  if ((q + 1) * L <= n) return reinterpret_cast<const VT*>(p)[q];
  zero16(v);
  TV* e = reinterpret_cast<TV*>(&v);
  for (int k = 0; k < L; ++k)
    if (q * L + k < n) e[k] = p[q * L + k];
  return v;
}

__device__ __forceinline__ float4 quotient16(const float4& x, float r, float rl) {
  return make_float4(quotient(x.x, r, rl), quotient(x.y, r, rl), quotient(x.z, r, rl), quotient(x.w, r, rl));
}
__device__ __forceinline__ double2 quotient16(const double2& x, double r, double rl) {
  return make_double2(quotient(x.x, r, rl), quotient(x.y, r, rl));
}

// T threads; a thread keeps U chunks of w in registers.  The basis vectors
// stream through a ring of RING halves (U / 2 chunks a thread) in shared
// memory: two whole vectors, or one and a half where that is all that fits.
// A slice longer than T U chunks (REST) leaves the remainder of w in global
// memory, BATCH chunks a thread in flight; that wants the registers, so few
// chunks stay in them (cycle of 8 directions at 8M / 16M / 40M FP32 elements:
// U = 8 and BATCH = 4 588 / 1736 / 4473 us, U = 18 and BATCH = 2 657 / 2035 /
// 5334).
constexpr int BATCH = 4;
template <int T, int U>
constexpr int column_ring = T * U <= 512 * 12 ? 4 : 3;

// the sentinel of an unwritten slot: a NaN that no addition produces
__device__ __forceinline__ double no_sum() { return __longlong_as_double(-1LL); }
__device__ __forceinline__ bool is_no_sum(double s) { return __double_as_longlong(s) == -1LL; }

// chunks of a run of FP32 products
template <int U>
constexpr int RUN = U < 10 ? 1 : U / 5;

// A thread's sum: FP64 in two halves, FP32 as hi + lo, lo the rounding errors of the
// joined runs (Knuth's TwoSum: six FP32 operations, where an addition in FP64
// would hold the warp's scheduler for 64 cycles)
template <typename TV>
struct Sum;
template <>
struct Sum<double> {
  double half[2] = {0.0, 0.0};
  __device__ __forceinline__ double total() const { return half[0] + half[1]; }
};
template <>
struct Sum<float> {
  float hi = 0.0f, lo = 0.0f;
  __device__ __forceinline__ void join(float run) {
    const float s = hi + run, b = s - hi;
    lo += (hi - (s - b)) + (run - b);
    hi = s;
  }
  __device__ __forceinline__ double total() const { return widen(hi) + widen(lo); }
};
// s + the products of chunks first .. first + H - 1 below used
template <int FIRST, int H, int RUN, typename VT, int U>
__device__ __forceinline__ void add_products(Sum<double>& s, const VT (&x)[U], const VT* v, int stride, int used) {
#pragma unroll
  for (int u = FIRST; u < FIRST + H; ++u)
    if (u < used) s.half[u >= U / 2] = dot16(x[u], v ? v[(u - FIRST) * stride] : x[u], s.half[u >= U / 2]);
}
template <int FIRST, int H, int RUN, typename VT, int U>
__device__ __forceinline__ void add_products(Sum<float>& s, const VT (&x)[U], const VT* v, int stride, int used) {
#pragma unroll
  for (int u0 = FIRST; u0 < FIRST + H; u0 += RUN)
    if (u0 < used) {
      float run = 0.0f;
#pragma unroll
      for (int u = u0; u < u0 + RUN && u < FIRST + H; ++u)
        if (u < used) run = dot16(x[u], v ? v[(u - FIRST) * stride] : x[u], run);
      if (u0 == 0)
        s.hi = run;
      else
        s.join(run);
    }
}

template <typename TV, int T, int U, bool REST>
__global__ void __launch_bounds__(T, 1)
    k_column(long n, long slice, TV* __restrict__ w, TV* __restrict__ V, long vs, int dir, int m, KrylovScalars* ks,
             double* __restrict__ slots, double* __restrict__ next_slots, int G, int spin_limit) {
  using VT = typename V16<TV>::T;
  using ST = std::conditional_t<REST, double, TV>;
  constexpr int L = V16<TV>::n;
  constexpr int H = U / 2, RING = column_ring<T, U>;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ ST sums[T];
  __shared__ TV lows[sizeof(TV) == 4 && !REST && T > 128 ? T : 1];  // the sums' lower parts
  __shared__ double warpSum[4];
  __shared__ double result;
  const int tid = threadIdx.x, lane = tid & 31;
  if ((int)blockIdx.x == G) {  // the helper: not part of the exchange
    if (tid == 0 && dir > 0) dev_hess(ks, dir - 1, m);
    return;
  }
  VT* buf = reinterpret_cast<VT*>(dyn) + tid;  // [RING][H][T]
  const long nv = (n + L - 1) / L;
  const long c0 = blockIdx.x * slice;
  const long c1 = c0 + slice < nv ? c0 + slice : nv;
  const long q0 = c0 + tid;  // this thread's chunks: q0 + u T, u < cnt
  const int cnt = q0 < c1 ? (int)min((c1 - q0 + T - 1) / T, (long)U) : 0;
  const long lastLeft = cnt ? (n - (q0 + (long)(cnt - 1) * T) * L) * (long)sizeof(TV) : 0;
  const int lastBytes = lastLeft < 16 ? (int)lastLeft : 16;  // the vector's end may fall inside a chunk
  // rows of chunks that hold any: a branch of the whole block, because an
  // FP64 instruction costs its 64 cycles with every lane predicated off too
  const int used = c1 > c0 ? (int)min((c1 - c0 + T - 1) / T, (long)U) : 0;
  const TV* src0 = V + q0 * L;
  // half vector hv of the stream (v_{hv / 2}, chunks of half hv % 2) into the ring
  auto issue = [&](int hv) {
    if (hv < 2 * (dir + 1)) {
      const TV* src = src0 + (size_t)(hv >> 1) * vs;
      VT* dst = buf + (hv % RING) * (H * T);
      const int first = (hv & 1) * H;
#pragma unroll
      for (int u = 0; u < H; ++u)
        if (first + u < used) {
          const int bytes = first + u < cnt - 1 ? 16 : (first + u == cnt - 1 ? lastBytes : 0);  // the rest is zero
          copy16(dst + u * T, bytes ? src + (size_t)(first + u) * T * L : V, bytes);
        }
    }
    copy_commit();
  };
#pragma unroll
  for (int hv = 0; hv < RING; ++hv) issue(hv);
  for (int s = tid; s < m + 2; s += T) next_slots[(size_t)s * G + blockIdx.x] = no_sum();
  if (ks->status) {
    copy_wait<0>();
    return;
  }
  VT x[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u < cnt)
      x[u] = load16(w, q0 + (long)u * T, n);
    else
      zero16(x[u]);
  }
  double total = 0.0;
  TV h = TV(0);
#pragma unroll 1
  for (int j = 0; j <= dir + 1; ++j) {
    if (j > 0) {
      // w -= h_{j-1} v_{j-1}; its halves of the ring take the next ones
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const VT* v = buf + ((2 * j - 2 + p) % RING) * (H * T);
#pragma unroll
        for (int u = 0; u < H; ++u)
          if (p * H + u < used) axpy16(x[p * H + u], h, v[u * T]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)  // read before they are refilled
        asm volatile("" ::"r"(*reinterpret_cast<const int*>(&x[u])) : "memory");
      issue(2 * j - 2 + RING);
      issue(2 * j - 1 + RING);
    }
    // the slice beyond the registers, while the refills are in flight: the
    // loads of BATCH chunks before their products; FP32 products of 8 chunks
    // at most add up in FP32
    double mine = 0.0;
    if constexpr (REST) {
      VT* w4 = reinterpret_cast<VT*>(w);
      const VT* vp = reinterpret_cast<const VT*>(V + (size_t)(j - 1) * vs);
      const VT* vn = reinterpret_cast<const VT*>(V + (size_t)j * vs);
      const bool back = j > 0, ahead = j <= dir;
      const long whole = min(c1, n / L);
      TV a = TV(0);
      int count = 0;
      long q = q0 + (long)U * T;
      for (; q + (BATCH - 1) * T < whole; q += BATCH * T) {
        VT y[BATCH], p[BATCH], v[BATCH];
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {
          y[k] = w4[q + k * T];
          if (back) p[k] = vp[q + k * T];
          if (ahead) v[k] = vn[q + k * T];
        }
#pragma unroll
        for (int k = 0; k < BATCH; ++k) {
          if (back) {
            axpy16(y[k], h, p[k]);
            w4[q + k * T] = y[k];
          }
          a = dot16(y[k], ahead ? v[k] : y[k], a);
        }
        if ((count += BATCH) == 8) {
          mine += widen(a);
          a = TV(0);
          count = 0;
        }
      }
      for (; q < c1; q += T) {
        VT y = load16(w, q, n);
        if (back) {
          axpy16(y, h, load16(V + (size_t)(j - 1) * vs, q, n));
          w4[q] = y;
        }
        a = dot16(y, ahead ? load16(V + (size_t)j * vs, q, n) : y, a);
      }
      mine += widen(a);
    }
    // the sum of this step: w . v_j, or |w|^2 at the end
    Sum<TV> a;
    if (j <= dir) {
      copy_wait<RING - 1>();
      add_products<0, H, RUN<U>>(a, x, buf + ((2 * j) % RING) * (H * T), T, used);
      copy_wait<RING - 2>();
      add_products<H, H, RUN<U>>(a, x, buf + ((2 * j + 1) % RING) * (H * T), T, used);
    } else {
      add_products<0, U, RUN<U>>(a, x, (const VT*)nullptr, T, used);
    }
    // block sum: four warps fold the threads' sums
    ST t;
    if constexpr (REST)
      t = mine + a.total();
    else if constexpr (sizeof(TV) == 8)
      t = a.total();
    else
      t = a.hi;
    if (T > 128) {
      sums[tid] = t;
      if constexpr (sizeof(TV) == 4 && !REST) lows[tid] = a.lo;
      __syncthreads();
    }
    if (tid < 128) {
      double s;
      if constexpr (sizeof(TV) == 4 && !REST) {
#pragma unroll
        for (int k = 1; k < T / 128; ++k) {
          a.join(sums[tid + 128 * k]);
          a.lo += lows[tid + 128 * k];
        }
        s = a.total();
      } else {
        s = widen(t);
#pragma unroll
        for (int k = 1; k < T / 128; ++k) s += widen(sums[tid + 128 * k]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) warpSum[tid >> 5] = s;
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    if (tid < 32) {
      double* row = slots + (size_t)j * G;
      if (lane == 0) {
        double s = (warpSum[0] + warpSum[1]) + (warpSum[2] + warpSum[3]);
        if (is_no_sum(s)) s = __longlong_as_double(0x7fffffffffffffffLL);
        asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(row + blockIdx.x), "d"(s) : "memory");
      }
      // every slot of the step, all loads of a poll in flight together
      double v[5];
      int it = 0;
      if (G > PAUSE_BLOCKS) __nanosleep(PAUSE_FIRST);
      while (true) {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const int b = lane + 32 * k;
          v[k] = 0.0;
          if (32 * k < G)
            asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v[k]) : "l"(row + (b < G ? b : 0)) : "memory");
        }
        bool ready = true;
#pragma unroll
        for (int k = 0; k < 5; ++k) ready = ready && !is_no_sum(v[k]);
        if (__all_sync(0xffffffffu, ready)) break;
        if ((++it & 63) == 0) {
          if (it > spin_limit && lane == 0) atomicOr(&ks->status, 8);
          if (__any_sync(0xffffffffu, it > spin_limit || (ld_relaxed_int(&ks->status) & 8))) break;
        }
        if (G > PAUSE_BLOCKS) __nanosleep(PAUSE_NEXT);
      }
#pragma unroll
      for (int k = 0; k < 5; ++k)
        if (lane + 32 * k >= G) v[k] = 0.0;
      double s = v[0];
      if (G > 32) s += v[1];
      if (G > 64) s += v[2] + v[3];
      if (G > 128) s += v[4];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) {
        result = s;
        if (blockIdx.x == 0) {
          if (j <= dir)
            ks->H[j * m + dir] = s;
          else if (dir >= 0)
            ks->nrm2[dir] = s;
        }
      }
    }
    __syncthreads();
    total = result;
    h = TV(total);
  }
  // the next basis vector (the last direction of a cycle needs none)
  if (dir + 1 < m) {
    const double beta = sqrt(total);
    if (dir < 0 && blockIdx.x == 0 && tid == 0) dev_beta0(ks, beta, m);
    // a zero start of a cycle is a breakdown (dev_beta0); a zero vector later on
    // is divided by its norm all the same, and the solve ends as not finite
    if (dir < 0 && !(beta > 0.0)) return;
    const TV b = TV(beta), rb = TV(1) / b, rl = rb * fma(-b, rb, TV(1));
    VT* out = reinterpret_cast<VT*>(V + (size_t)(dir + 1) * vs);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < cnt) out[q0 + (long)u * T] = quotient16(x[u], rb, rl);
    if constexpr (REST) {
      for (long q = c0 + (long)U * T + tid; q < c1; q += T) out[q] = quotient16(load16(w, q, n), rb, rl);
    }
  }
}

template <typename TV, int T, int U, bool REST>
void launch_column(Handle& h, int blocks, long slice, long n, TV* w, TV* V, long vs, int dir, int m, double* slots,
                   double* next) {
  auto kern = k_column<TV, T, U, REST>;
  const size_t smem = (size_t)column_ring<T, U> * (U / 2) * T * 16;
  ICS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  KrylovScalars* ks = h.ks;
  int spin = h.columnProbe ? h.columnProbe : COLUMN_SPIN_LIMIT;
  void* args[] = {&n, &slice, &w, &V, &vs, &dir, &m, &ks, &slots, &next, &blocks, &spin};
  // with the probe the last block of the exchange (and the helper) never runs
  const int grid = h.columnProbe && blocks > 1 ? blocks - 1 : blocks + 1;
  ICS_LAUNCH(h, ICS_K_MGS,
             ICS_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(T), args, smem, h.stream)));
}

// the instance with the fewest chunks per thread that holds a slice: chunks a
// thread does not use would still cost their FP64 instructions
template <typename TV, int U, typename... Args>
void launch_sized(Handle& h, int blocks, long slice, Args... args) {
  if constexpr (U <= 18) {
    if (slice <= 128L * U && U <= 4)
      launch_column<TV, 128, U, false>(h, blocks, slice, args...);
    else if (slice <= 512L * U)
      launch_column<TV, 512, U, false>(h, blocks, slice, args...);
    else
      launch_sized<TV, U + 2>(h, blocks, slice, args...);
  } else {
    launch_column<TV, 512, 8, true>(h, blocks, slice, args...);
  }
}

template <typename TV>
void column_t(Handle& h, long n, TV* w, TV* V, long vs, int dir, int m) {
  constexpr int L = V16<TV>::n;
  const long nv = (n + L - 1) / L;
  // SMALL_GRID blocks while their cheaper exchange outweighs the work that
  // more would take over (a column cycle of 8 directions, us: FP64 50k
  // elements 117 against 130, 983k 365 against 349; FP32 586k 145 against 152,
  // 1.1M 163 both, 5.2M 390 against 318), else one per SM with the helper on
  // an SM of its own; no more than give every block 128 chunks
  const int most = std::min(h.sms - 1, MAX_GRID);
  const long large = sizeof(TV) == 4 ? 2000000 : 300000;
  const int G = (int)std::max(1L, std::min((long)(n > large ? most : std::min(most, SMALL_GRID)), (nv + 127) / 128));
  const long slice = (nv + G - 1) / G;
  // three sets of slots: two alternate over the directions, one is the
  // cycle start's; a column resets the set of the one that follows it
  const size_t set = (size_t)(m + 2) * G;
  auto at = [&](int d) { return h.colSlots + set * (d < 0 ? 2 : (d & 1)); };
  launch_sized<TV, 2>(h, G, slice, n, w, V, vs, dir, m, at(dir), at(dir + 1 < m ? dir + 1 : -1));
}

}  // namespace

size_t column_slot_words() { return 3ull * (MAX_DIRS + 2) * MAX_GRID; }

void column_reset(Handle& h, int m) {
  ICS_CUDA(cudaMemsetAsync(h.colSlots, 0xff, 3ull * (m + 2) * MAX_GRID * sizeof(double), h.stream));
}

void krylov_column(Handle& h, bool fp32, long n, void* w, void* V, long vs, int dir, int m) {
  if (fp32)
    column_t<float>(h, n, (float*)w, (float*)V, vs, dir, m);
  else
    column_t<double>(h, n, (double*)w, (double*)V, vs, dir, m);
}

}  // namespace ics
