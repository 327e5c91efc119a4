// One-launch Krylov iterations: the CG loop of one system inside a single
// kernel, the row slices of the SELL matrix divided over the thread blocks of
// a group that stays resident for the whole loop.
//
// What bounds it.  As a graph of three kernels an iteration of a system that
// fits the L2 cost 21 us at 961 unknowns and 26 us at 129k: every kernel
// waited for its flags and scalars, re-read the vectors of its rows, and ended
// in a last-block reduction, each a chain of memory round trips and of FP64
// adds (64 cycles apiece).  Here
//   - a thread block keeps the same rows for the whole solve: x, r, p, q and
//     the preconditioner stay in shared memory, and the matrix too when it
//     fits (MS); only what is gathered goes through global memory;
//   - the sums go thread -> warp -> block -> group, and one warp of every
//     block forms alpha, beta and the convergence test from the group totals
//     (the same partials in the same order: the same bits in every block);
//   - x is advanced between the arrival at and the wait for the second sum.
// Per iteration, quadratic heat, FP64 and FP32 (graphs, then one launch):
//       961 unknowns  21.3 ->  6.3 us   25.8 ->  9.6 us (12 replacements incl.)
//     14161           21.1 -> 10.1      21.9 ->  7.5
//    128881           26.2 -> 13.8      22.2 ->  9.4
//    358801           40.2 -> 23.2      32.0 -> 13.9
//    808201           62.7 -> 46.6      45.9 -> 21.1
// MINRES (Taylor-Hood cavity) 27.2 -> 12.5 us at 9026 unknowns.  What is left
// is the barriers (about 4 us of the 13.8) and the FP64 unit (6 us of them).
// Two groups are provided:
//   ClusterGroup  one cluster of up to 16 blocks: sums through distributed
//                 shared memory, the hardware cluster barrier (0.2-0.3 us);
//   GridGroup     one block per SM, launched cooperatively: an arrival counter
//                 in global memory (1.1 us per barrier at 152 blocks).  Every
//                 wait is bounded; a wait that runs out marks the error word
//                 and ends the kernel.
// FP64 work grows with 1 / blocks, so a cluster of 16 SMs serves systems up to
// 16k unknowns in FP64 (at 14k: 10.1 us, at 22k in a grid 9.2) and, bound by
// its barriers instead, 32k in FP32.
#include <cooperative_groups.h>

#include <algorithm>

#include "krylov.cuh"

namespace elfel {

namespace {

namespace cg = cooperative_groups;

constexpr int kRT = kRunThreads;
constexpr int kRW = kRT / 32;
constexpr int kRunPart = 3 * kRT + 16;  // doubles of shared memory for the block sums
constexpr unsigned kRunSpins = 1u << 22;  // polls of the arrival counter, about a second

// Sums.  The FP64 unit of an SM sub-partition takes a warp instruction every
// 64 cycles whatever its active lanes, so what a sum costs is the number of
// FP64 instructions one after another: they are spread over warps 0-3 (one
// per sub-partition), and NV values share a warp, L lanes each.
__host__ __device__ constexpr int sum_groups(int nv) { return nv == 1 ? 1 : nv == 2 ? 2 : 4; }

__device__ __forceinline__ void quad_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// s of each lane added over its group of L lanes (a power of two).
template <int L>
__device__ __forceinline__ double lanes_sum(double s) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// 1 / x by Newton's iteration from the hardware's 20-bit estimate (four FP64
// operations; the compiler's division takes about twelve, 64 cycles each).
// x of extreme exponent goes through the division.
__device__ __forceinline__ double fast_rcp(double x) {
  const int e = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  if (e < 60 || e > 1980) return 1.0 / x;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// a / x, y = fast_rcp(x): the quotient corrected by its remainder.
__device__ __forceinline__ double fast_div(double a, double x, double y) {
  const double q = a * y;
  return fma(fma(-x, q, a), y, q);
}

// x > 0 and finite, a <= b, a < b for nonnegative a, b (and NaN above all of
// them): integer comparisons, which leave the FP64 unit alone.
__device__ __forceinline__ bool pos_finite(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b < 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool finite(double x) {
  return (__double_as_longlong(x) & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool le_pos(double a, double b) { return __double_as_longlong(a) <= __double_as_longlong(b); }
__device__ __forceinline__ bool lt_pos(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }

// The sums of warps 0-3 (value g in the lanes of group g) to totals: tot[k]
// in every lane of warp 0.  wsum: 16 doubles of shared memory.
template <int NV>
__device__ __forceinline__ void quad_total(double s, double* wsum, double (&tot)[NV]) {
  constexpr int L = 32 / sum_groups(NV);
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / L;
  if (lane % L == 0 && g < NV) wsum[g * 4 + wid] = s;
  quad_barrier();
  if (wid == 0) {
    const double x = lanes_sum<4>(lane < 4 * NV ? wsum[lane] : 0.0);
#pragma unroll
    for (int k = 0; k < NV; ++k) tot[k] = __shfl_sync(0xffffffffu, x, 4 * k);
  }
}

// Groups.  A sum over the group's blocks: warp 0 publishes the block's NV
// values (the same in every lane), all threads call arrive and wait, warps 0-3
// collect the totals (valid in warp 0; collect alternates the buffers).
// arrive/wait are a barrier of the group which also makes the blocks' earlier
// global writes visible; wait returns false in warp 0 when it ran out.
struct ClusterGroup {
  cg::cluster_group cl;
  int n, rank, par;
  struct Shared {
    double part[2][3][16];
  };
  Shared* sh;
  __device__ ClusterGroup(const RunGroup&, Shared* s) : cl(cg::this_cluster()), par(0), sh(s) {
    n = (int)cl.num_blocks();
    rank = (int)cl.block_rank();
    cl.sync();  // every block of the cluster runs: its shared memory may be written
  }
  template <int NV>
  __device__ __forceinline__ void publish(const double (&v)[NV]) {
    const int lane = threadIdx.x & 31;
    if (lane < n) {
#pragma unroll
      for (int k = 0; k < NV; ++k) *cl.map_shared_rank(&sh->part[par][k][rank], lane) = v[k];
    }
  }
  __device__ __forceinline__ void arrive(int) { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
  __device__ __forceinline__ bool wait(int) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  template <int NV>
  __device__ __forceinline__ void collect(int wid, double*, double (&t)[NV]) {
    constexpr int L = 32 / sum_groups(NV);
    if (wid == 0) {
      const int lane = threadIdx.x & 31, g = lane / L, l = lane % L;
      double s = 0.0;
      if (g < NV) {
        s = l < n ? sh->part[par][g][l] : 0.0;
        if (L < 16 && l + L < n) s += sh->part[par][g][l + L];
      }
      s = lanes_sum<L>(s);
#pragma unroll
      for (int k = 0; k < NV; ++k) t[k] = __shfl_sync(0xffffffffu, s, k * L);
    }
    par ^= 1;
  }
  // barrier that ends an iteration: the blocks' slices of the direction are visible
  __device__ __forceinline__ void arrive_halo(int wid) { arrive(wid); }
  __device__ __forceinline__ bool wait_halo(int wid) { return wait(wid); }
  static constexpr bool kCluster = true;
};

struct GridGroup {
  RunGroup g;
  int n, par;
  unsigned target, epoch;
  int2 halo;  // blocks whose rows this block's columns lie in
  struct Shared {
    int dummy;
  };
  __device__ GridGroup(const RunGroup& rg, Shared*) : g(rg), par(0), target(0), epoch(0) {
    n = (int)gridDim.x;
    halo = rg.neighbours ? rg.halo[blockIdx.x] : make_int2(0, 0);
  }
  template <int NV>
  __device__ __forceinline__ void publish(const double (&v)[NV]) {
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) __stcg(g.slots + ((size_t)par * 3 + k) * kRunMaxBlocks + blockIdx.x, v[k]);
    }
  }
  // Warp 0 arrives for the block: a block barrier comes before, so that the
  // other warps' writes do too.
  __device__ __forceinline__ void arrive(int) {
    target += (unsigned)n;
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(g.words, 1u);
    }
  }
  // Polls word w until it has reached v (warp 0, by lane; inactive lanes pass).
  __device__ __forceinline__ bool poll(const unsigned* w, unsigned v, bool active) {
    bool ok = true, here = !active;
    for (unsigned spins = 0; !__all_sync(0xffffffffu, here); ++spins) {
      if (!here) {
        unsigned x;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(w) : "memory");
        here = (int)(x - v) >= 0;
      }
      const bool out = spins > kRunSpins || ((spins & 1023u) == 1023u && *(volatile unsigned*)(g.words + 1));
      if (__any_sync(0xffffffffu, out)) {
        if (threadIdx.x == 0) atomicExch(g.words + 1, 1u);
        ok = false;
        break;
      }
    }
    __threadfence();
    return ok;
  }
  __device__ __forceinline__ bool wait(int wid) { return wid ? true : poll(g.words, target, threadIdx.x == 0); }
  template <int NV>
  __device__ __forceinline__ void collect(int wid, double* wsum, double (&t)[NV]) {
    if (wid < 4) {
      quad_barrier();  // warp 0 has seen every block's arrival
      constexpr int L = 32 / sum_groups(NV), Q = kRunMaxBlocks / 4;
      const int lane = threadIdx.x & 31, gr = lane / L, l = lane % L;
      const double* p = g.slots + ((size_t)par * 3 + gr) * kRunMaxBlocks + wid * Q;
      double w[(Q + L - 1) / L];
#pragma unroll
      for (int j = 0; j < (Q + L - 1) / L; ++j) {
        const int b = l + j * L;
        w[j] = gr < NV && b < Q && wid * Q + b < n ? __ldcg(p + b) : 0.0;
      }
      double s = w[0];
#pragma unroll
      for (int j = 1; j < (Q + L - 1) / L; ++j) s += w[j];
      quad_total<NV>(lanes_sum<L>(s), wsum, t);
    }
    par ^= 1;
  }
  // The barrier that ends an iteration, before the next gathers: where a
  // block gathers from at most 32 blocks around its own it waits for those
  // alone (a flag each); a block rewrites its rows of the direction only after
  // two more sums, which every block enters after its gathers.
  __device__ __forceinline__ void arrive_halo(int wid) {
    if (!g.neighbours) {
      arrive(wid);
      return;
    }
    ++epoch;
    if (threadIdx.x == 0) {
      __threadfence();
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(g.words + kRunFlag0 + blockIdx.x * kRunFlagStride), "r"(epoch)
                   : "memory");
    }
  }
  __device__ __forceinline__ bool wait_halo(int wid) {
    if (!g.neighbours) return wait(wid);
    if (wid) return true;
    const int b = halo.x + (int)threadIdx.x;
    return poll(g.words + kRunFlag0 + b * kRunFlagStride, epoch, b <= halo.y);
  }
  static constexpr bool kCluster = false;
};

// The block's sums of the threads' values, in every lane of warp 0 (which
// has room for 3 * kRT doubles in part and 16 in wsum).  FP32 values add
// within the warp in FP32 first; FP64 values go to shared memory as they are.
template <int NV, typename T>
__device__ __forceinline__ void block_sums(T (&v)[NV], double* part, double* wsum, double (&tot)[NV]) {
  constexpr int L = 32 / sum_groups(NV);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane / L, l = lane % L;
  if (sizeof(T) == 4) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if (lane == 0) part[k * kRW + wid] = (double)v[k];
    }
    __syncthreads();
    if (wid == 0) {
      double s = 0.0;
      if (g < NV && l < kRW) {
        s = part[g * kRW + l];
#pragma unroll
        for (int j = 1; j * L < kRW; ++j) s += part[g * kRW + l + j * L];
      }
      s = lanes_sum<L>(s);
#pragma unroll
      for (int k = 0; k < NV; ++k) tot[k] = __shfl_sync(0xffffffffu, s, k * L);
    }
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k) part[k * kRT + threadIdx.x] = (double)v[k];
    __syncthreads();
    if (wid < 4) {
      double s = 0.0;
      if (g < NV) {
        const double* p = part + g * kRT + wid * (kRT / 4) + l;
        s = p[0];
#pragma unroll
        for (int j = 1; j < kRT / 4 / L; ++j) s += p[j * L];
      }
      quad_total<NV>(lanes_sum<L>(s), wsum, tot);
    }
  }
}

// A gathered entry of the direction: x[c], or z[c] + beta x[c] when the new
// direction is formed where it is gathered (TWO).  Plain loads: other blocks
// rewrite both between the group's barriers, whose acquire refreshes L1.
template <typename T>
__device__ __forceinline__ T axpy(T b, T x, T z) {
  return sizeof(T) == 4 ? (T)fmaf((float)b, (float)x, (float)z) : (T)fma((double)b, (double)x, (double)z);
}
template <typename T, bool TWO>
__device__ __forceinline__ T gather(const T* x, const T* z, T beta, int c) {
  return TWO ? axpy<T>(beta, x[c], z[c]) : x[c];
}

// U entries of a row from entry j on: the columns and values of all of them
// are loaded before the gathers, so that U gathers are in flight.  With TAIL
// the entries beyond w are left out (w is the same in all lanes).
template <typename T, bool D16, bool DIFF, bool MS, bool TWO, int U, bool TAIL, typename C>
__device__ __forceinline__ void run_part(const T* v, const C* cols, int base, int j, int w, int64_t row, const T* x,
                                         const T* z, T beta, T xi, T (&a)[4]) {
  int cc[U];
  T vv[U], xx[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (!TAIL || j + u < w) {
      const C c = MS ? cols[base + 32 * (j + u)] : __ldcg(cols + base + 32 * (j + u));
      cc[u] = D16 ? (int)row + (int)c : (int)c;
    }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (!TAIL || j + u < w) vv[u] = MS ? v[base + 32 * (j + u)] : __ldcg(v + base + 32 * (j + u));
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (!TAIL || j + u < w) xx[u] = xterm<T, DIFF>(gather<T, TWO>(x, z, beta, cc[u]), cc[u], row, xi);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (!TAIL || j + u < w) a[u & 3] += vv[u] * xx[u];
}

// One row of a slice, the matrix in shared memory (MS: v, cols and base are
// the block's copies) or in global memory.  FP32 takes a predicated tail; an
// FP64 multiply-add costs the same left out by a predicate, so FP64 takes the
// tail in parts of 4, 2 and 1 (N = 180 quadratic heat: 8.0k cycles a product
// with the predicated tail, 6.4k so).
template <typename T, bool D16, bool DIFF, bool MS, bool TWO, typename C>
__device__ __forceinline__ T run_row(const T* v, const C* cols, int base, int w, int64_t row, const T* x, const T* z,
                                     T beta, T xi) {
  T a[4] = {0, 0, 0, 0};
  constexpr int U = sizeof(T) == 4 ? 10 : 8;
  int j = 0;
#define RUN_PART(n, tail) run_part<T, D16, DIFF, MS, TWO, n, tail, C>(v, cols, base, j, w, row, x, z, beta, xi, a)
  for (; j + U <= w; j += U) RUN_PART(U, false);
  if (sizeof(T) == 4) {
    if (j < w) RUN_PART(U, true);
  } else {
    if ((w - j) & 4) {
      RUN_PART(4, false);
      j += 4;
    }
    if ((w - j) & 2) {
      RUN_PART(2, false);
      j += 2;
    }
    if ((w - j) & 1) RUN_PART(1, false);
  }
#undef RUN_PART
  return (a[0] + a[1]) + (a[2] + a[3]);
}

// What warp 0 tells the block after a sum.
struct RunMsg {
  double c[5];
  int stop;  // leave the loop: 1 at the iteration's end, 2 at once (a wait ran out)
};

// The block's part of the system: its slices, and the matrix (in shared
// memory when MS) with its slice bases and widths.
template <typename T, bool D16, bool MS>
struct RunRows {
  typedef typename ColType<D16>::type C;
  int64_t row0;
  int nsl, nloc;
  const T* mv;
  const C* mc;
  const int2* sbw;
  // sbw_sh: room for spb slices, followed by the matrix (MS)
  __device__ __forceinline__ RunRows(const SellView& A, const T* v, int spb, int max_entries, int2* sbw_sh) {
    const int tid = threadIdx.x;
    const int64_t s0 = (int64_t)blockIdx.x * spb;
    nsl = (int)max((int64_t)0, min((int64_t)spb, A.nslices - s0));
    row0 = s0 * 32;
    nloc = nsl > 0 ? (int)min((int64_t)nsl * 32, A.nrows - row0) : 0;
    const int64_t e0 = nsl > 0 ? A.sptr[s0] : 0;
    const C* gc = reinterpret_cast<const C*>(D16 ? (const void*)A.d16 : (const void*)A.c32) + e0;
    const T* gv = v + e0;
    for (int s = tid; s < nsl; s += kRT) sbw_sh[s] = make_int2((int)(A.sptr[s0 + s] - e0), A.sw[s0 + s]);
    sbw = sbw_sh;
    mv = gv;
    mc = gc;
    if (MS) {
      T* sv = reinterpret_cast<T*>(sbw_sh + spb);
      C* sc = reinterpret_cast<C*>(sv + max_entries);
      const int ne = nsl > 0 ? (int)(A.sptr[s0 + nsl] - e0) : 0;
      for (int k = tid; k < ne; k += kRT) {
        sv[k] = gv[k];
        sc[k] = gc[k];
      }
      mv = sv;
      mc = sc;
    }
  }
  // The n-th slice of a warp.  Within a window of 8 slices the long rows come
  // first (sigma = 256): the windows are handed out rotated by two, so that
  // the four sub-partitions get as many long slices each.
  __device__ __forceinline__ static int slice(int wid, int n) {
    const int win = n * (kRW / 8) + (wid >> 3);
    return win * 8 + ((wid - 2 * win) & 7);
  }
  // (A p)_i of local row i in slice s; p = x, or z + beta x (TWO); xi: p_i
  template <bool DIFF, bool TWO>
  __device__ __forceinline__ T row(int s, int i, const T* x, const T* z, T beta, T xi) const {
    const int2 bw = sbw[s];
    return run_row<T, D16, DIFF, MS, TWO, C>(mv, mc, bw.x + (i & 31), bw.y, row0 + i, x, z, beta, xi);
  }
};

// CG on the permuted system.  IR: the FP32 recurrence of the refinement
// (difference form, flexible step, Polak-Ribiere beta; stops for a residual
// replacement), else FP64 Jacobi PCG.  The recurrences and stopping rules are
// those of the graph kernels (sell_cg_spmv_k, cg_update_k, cg_p_k).
//
// The direction p = z + beta p needs beta, which needs every block: written
// out and gathered after a third barrier; or (TWO) z is written before the
// second sum, and the product gathers z + beta p with the p of the iteration
// before, one multiply-add more per entry instead of the barrier.  p then
// alternates between two buffers.
template <typename T, bool D16, bool IR, bool MS, bool TWO, class Group>
__global__ void __launch_bounds__(kRT, 1) cg_run_k(const CgRun<T> a, const RunGroup rg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ typename Group::Shared gsh;
  __shared__ RunMsg msg;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  double* part = reinterpret_cast<double*>(smem);
  double* wsum = part + 3 * kRT;
  T* sx = reinterpret_cast<T*>(part + kRunPart);
  const int ld = a.spb * 32;
  T *sr = sx + ld, *sp = sr + ld, *sq = sp + ld, *sd = sq + ld;
  const RunRows<T, D16, MS> R(a.A, a.v, a.spb, a.max_entries, reinterpret_cast<int2*>(sd + ld));
  for (int i = tid; i < R.nloc; i += kRT) {
    sx[i] = a.x[R.row0 + i];
    sr[i] = a.r[R.row0 + i];
    const T p = a.p[R.row0 + i];
    sp[i] = TWO ? 0 : p;
    if (TWO) sq[i] = p;  // the first direction is z + 0 p
    sd[i] = a.dinv[R.row0 + i];
  }
  // the loop's scalars (warp 0 uses them)
  double rz = a.scal[S_RZ], rr = a.scal[S_RR], pq = 0.0, alpha = 0.0, beta = 0.0, inv_rz = 1.0 / rz;
  const double thr = a.scal[S_TOL2] * (IR ? a.scal[S_BN2S] : a.scal[S_BN2]);
  const double delta2 = IR ? a.scal[S_DELTA] * a.scal[S_DELTA] : 0.0;
  double rmax2 = a.scal[S_RMAX] * a.scal[S_RMAX];  // the largest r.r since the last replacement
  double low2 = delta2 * rmax2;
  int it = a.flags[F_ITER], done = 0, conv = 0, ru = 0, brk = a.flags[F_BRK];
  const int maxit = a.flags[F_MAXIT];
  Group grp(rg, &gsh);
  __syncthreads();

  // what the product gathers: (z, p of the iteration before), first (p, p) with beta = 0
  const T *zg = a.p, *pold = a.p;
  T* pnew = TWO ? a.p2 : a.p;
  T be = 0;
  for (int k = 0; k < a.max_iters; ++k) {
    // (p = z + beta p) q = A p; p.q (and r.p) -> alpha
    constexpr int N1 = IR ? 2 : 1;
    T d1[N1] = {};
    for (int n = 0; n * kRW < R.nsl; ++n) {
      const int s = R.slice(wid, n);
      const int i = s * 32 + lane;
      if (i < R.nloc) {
        T pi = sp[i];
        if (TWO) {
          pi = axpy<T>(be, pi, sq[i]);
          sp[i] = pi;
          pnew[R.row0 + i] = pi;
        }
        const T acc = R.template row<IR, TWO>(s, i, pold, zg, be, pi);
        sq[i] = acc;
        d1[0] += acc * pi;
        if (IR) d1[N1 - 1] += sr[i] * pi;
      }
    }
    double t1[N1];
    block_sums<N1>(d1, part, wsum, t1);
    if (wid == 0) grp.publish(t1);
    grp.arrive(wid);
    bool ok = grp.wait(wid);
    grp.collect(wid, wsum, t1);
    if (wid == 0) {
      pq = t1[0];
      alpha = pos_finite(pq) ? fast_div(IR ? t1[N1 - 1] : rz, pq, fast_rcp(pq)) : 0.0;
      if (lane == 0) {
        msg.c[0] = alpha;
        msg.stop = ok ? 0 : 2;
      }
    }
    __syncthreads();
    if (msg.stop) break;
    // r -= alpha q, z = D r (kept in q); r.z, r.r (and z.r_old) -> beta
    constexpr int N2 = IR ? 3 : 2;
    const T al = (T)msg.c[0];
    T d2[N2] = {};
    for (int i = tid; i < R.nloc; i += kRT) {
      const T ro = sr[i];
      const T ri = ro - al * sq[i];
      sr[i] = ri;
      const T zi = sd[i] * ri;
      sq[i] = zi;
      if (TWO) a.z[R.row0 + i] = zi;
      d2[0] += ri * zi;
      d2[1] += ri * ri;
      if (IR) d2[N2 - 1] += zi * ro;
    }
    double t2[N2];
    block_sums<N2>(d2, part, wsum, t2);
    if (wid == 0) grp.publish(t2);
    grp.arrive(wid);
    for (int i = tid; i < R.nloc; i += kRT) sx[i] += al * sp[i];
    if (wid == 0) inv_rz = fast_rcp(rz);
    ok = grp.wait(wid);
    grp.collect(wid, wsum, t2);
    if (wid == 0) {
      const double rzn = t2[0];
      rr = t2[1];
      beta = (IR ? rzn - t2[N2 - 1] : rzn) * inv_rz;
      rz = rzn;
      ++it;
      conv = le_pos(rr, thr);
      // breakdown: p.Ap not positive or not finite
      const bool bad = !pos_finite(pq) || !finite(rz) || !finite(rr);
      if (!IR) {
        done = conv || bad || it >= maxit;
        conv = conv && !bad;
      } else if (bad) {
        brk = 1;  // replace the residual and restart the direction from it
        ru = 1;
      } else {
        if (lt_pos(rmax2, rr)) {
          rmax2 = rr;
          low2 = delta2 * rmax2;
        }
        if (conv) brk = 2;  // spent directions: the replacement restarts from p = z
        ru = conv || it >= maxit || lt_pos(rr, low2);
      }
      if (lane == 0) {
        msg.c[0] = beta;
        msg.stop = !ok ? 2 : (done || ru) ? 1 : 0;
      }
    }
    __syncthreads();
    const int stop = msg.stop;
    if (stop == 2) break;
    be = (T)msg.c[0];
    if (TWO) {
      if (stop) break;
      zg = a.z;
      pold = pnew;
      pnew = pnew == a.p2 ? a.p : a.p2;
      continue;
    }
    for (int i = tid; i < R.nloc; i += kRT) {
      const T pn = axpy<T>(be, sp[i], sq[i]);
      sp[i] = pn;
      pnew[R.row0 + i] = pn;
    }
    if (stop) break;
    // the new direction is complete before the next gathers
    if (!Group::kCluster) __syncthreads();
    grp.arrive_halo(wid);
    ok = grp.wait_halo(wid);
    if (!Group::kCluster) {
      if (tid == 0) msg.stop = ok ? 0 : 2;
      __syncthreads();
      if (msg.stop) break;
    }
  }
  __syncthreads();
  for (int i = tid; i < R.nloc; i += kRT) {
    a.x[R.row0 + i] = sx[i];
    a.r[R.row0 + i] = sr[i];
    if (TWO) a.p[R.row0 + i] = axpy<T>(be, sp[i], sq[i]);
  }
  if (blockIdx.x == 0 && tid == 0) {
    a.scal[S_RZ] = rz;
    a.scal[S_RR] = rr;
    a.scal[S_PQ] = pq;
    a.scal[S_ALPHA] = alpha;
    a.scal[S_BETA] = beta;
    a.scal[S_RMAX] = sqrt(rmax2);
    a.flags[F_ITER] = it;
    if (!IR) {
      a.flags[F_DONE] = done;
      a.flags[F_CONV] = conv;
    }
    a.flags[F_RU] = ru;
    a.flags[F_BRK] = brk;
  }
  if (Group::kCluster) {  // no block leaves while another may still write its shared memory
    grp.arrive(wid);
    grp.wait(wid);
  }
}

// Preconditioned MINRES, the three steps of mr_spmv_k / mr_vec_k / mr_upd_k /
// mr_tail_k.  The scalar chain of a step (two square roots and five
// divisions) runs in warp 0 with the divisions side by side in its lanes; w
// and x are advanced between the arrival at and the wait for the barrier that
// ends the iteration.
template <typename T, bool D16, bool MS, class Group>
__global__ void __launch_bounds__(kRT, 1) mr_run_k(const MrRun<T> a, const RunGroup rg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ typename Group::Shared gsh;
  __shared__ RunMsg msg;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  double* part = reinterpret_cast<double*>(smem);
  double* wsum = part + 3 * kRT;
  T* sx = reinterpret_cast<T*>(part + kRunPart);
  const int ld = a.spb * 32;
  T *sz = sx + ld, *sq = sz + ld, *sm = sq + ld, *sv = sm + ld, *svm = sv + ld, *sw = svm + ld, *swm = sw + ld;
  const RunRows<T, D16, MS> R(a.A, a.v, a.spb, a.max_entries, reinterpret_cast<int2*>(swm + ld));
  const int64_t r0 = R.row0;
  for (int i = tid; i < R.nloc; i += kRT) {
    sx[i] = a.x[r0 + i];
    sz[i] = a.z[r0 + i];
    sm[i] = a.minv[r0 + i];
    sv[i] = a.vj[r0 + i];
    svm[i] = a.vjm[r0 + i];
    sw[i] = a.wj[r0 + i];
    swm[i] = a.wjm[r0 + i];
  }
  double gam = a.scal[S_GAM], gamp = a.scal[S_GAMP], c = a.scal[S_C], cp = a.scal[S_CP], s = a.scal[S_S],
         sp = a.scal[S_SP], eta = a.scal[S_ETA];
  const double stop_at = sqrt(a.scal[S_TOL2]) * a.scal[S_ETA0];
  double bcoef = gamp > 0.0 ? gam / gamp : 0.0;
  int it = a.flags[F_ITER], done = a.flags[F_DONE], conv = a.flags[F_CONV];
  const int maxit = a.flags[F_MAXIT];
  Group grp(rg, &gsh);
  __syncthreads();

  for (int k = 0; k < a.max_iters; ++k) {
    if (done && k == 0) break;  // nothing to do (zero right-hand side)
    // q = A z, delta = q.z
    T d1[1] = {0};
    for (int n = 0; n * kRW < R.nsl; ++n) {
      const int sl = R.slice(wid, n);
      const int i = sl * 32 + lane;
      if (i < R.nloc) {
        const T zi = sz[i];
        const T acc = R.template row<false, false>(sl, i, a.z, a.z, (T)0, zi);
        sq[i] = acc;
        d1[0] += acc * zi;
      }
    }
    double t[1];
    block_sums<1>(d1, part, wsum, t);
    if (wid == 0) grp.publish(t);
    grp.arrive(wid);
    bool ok = grp.wait(wid);
    double delta = 0.0;
    grp.collect(wid, wsum, t);
    if (wid == 0) {
      delta = t[0];
      if (lane == 0) {
        msg.c[0] = delta / gam;
        msg.c[1] = bcoef;
        msg.stop = ok ? 0 : 2;
      }
    }
    __syncthreads();
    if (msg.stop) break;
    // v' = q - (delta/gam) v_j - (gam/gamp) v_{j-1}, z' = M v' (in q), gamn^2 = z'.v'
    const T ca = (T)msg.c[0], cb = (T)msg.c[1];
    T d2[1] = {0};
    for (int i = tid; i < R.nloc; i += kRT) {
      const T vv = sq[i] - ca * sv[i] - cb * svm[i];
      svm[i] = vv;
      const T zz = sm[i] * vv;
      sq[i] = zz;
      d2[0] += zz * vv;
    }
    block_sums<1>(d2, part, wsum, t);
    if (wid == 0) grp.publish(t);
    grp.arrive(wid);
    ok = grp.wait(wid);
    grp.collect(wid, wsum, t);
    if (wid == 0) {
      const double gamn = sqrt(fmax(t[0], 0.0));
      const double a0 = c * delta - cp * s * gam;
      const double a1 = sqrt(a0 * a0 + gamn * gamn);
      const double a2 = s * delta + cp * c * gam;
      const double a3 = sp * gam;
      // a0 / a1, gamn / a1, 1 / a1, 1 / gamn, gamn / gam: one division in five lanes
      const double num = lane == 0 ? a0 : (lane == 1 || lane == 4) ? gamn : 1.0;
      const double den = lane < 3 ? a1 : lane == 4 ? gam : gamn;
      const double qd = num / den;
      const double cn = __shfl_sync(0xffffffffu, qd, 0), sn = __shfl_sync(0xffffffffu, qd, 1);
      const double ia1 = __shfl_sync(0xffffffffu, qd, 2), ig = __shfl_sync(0xffffffffu, qd, 3);
      const double bn = __shfl_sync(0xffffffffu, qd, 4);
      const double ce = cn * eta;
      cp = c;
      c = cn;
      sp = s;
      s = sn;
      gamp = gam;
      gam = gamn;
      bcoef = gamp > 0.0 ? bn : 0.0;
      eta = -s * eta;
      ++it;
      conv = fabs(eta) <= stop_at;
      done = conv || it >= maxit || gamn == 0.0;
      conv = conv || gamn == 0.0;
      if (lane == 0) {
        msg.c[0] = gamn > 0.0 ? ig : 0.0;
        msg.c[1] = a3;
        msg.c[2] = a2;
        msg.c[3] = ia1;
        msg.c[4] = ce;
        msg.stop = !ok ? 2 : done ? 1 : 0;
      }
    }
    __syncthreads();
    const int stop = msg.stop;
    if (stop == 2) break;
    const T zs = (T)msg.c[0], ca3 = (T)msg.c[1], ca2 = (T)msg.c[2], cia = (T)msg.c[3], cce = (T)msg.c[4];
    // w' = (z - a3 w_{j-1} - a2 w_j) / a1, x += c eta w', z = z' / gamn
    for (int i = tid; i < R.nloc; i += kRT) {
      const T zi = sz[i], zn = sq[i] * zs;
      sz[i] = zn;
      a.z[r0 + i] = zn;
      sq[i] = zi;
    }
    if (!Group::kCluster) __syncthreads();
    if (!stop) grp.arrive_halo(wid);
    for (int i = tid; i < R.nloc; i += kRT) {
      const T w = (sq[i] - ca3 * swm[i] - ca2 * sw[i]) * cia;
      swm[i] = w;
      sx[i] += cce * w;
    }
    T* tv = sv;
    sv = svm;
    svm = tv;
    T* tw = sw;
    sw = swm;
    swm = tw;
    if (stop) break;
    ok = grp.wait_halo(wid);
    if (!Group::kCluster) {
      if (tid == 0) msg.stop = ok ? 0 : 2;
      __syncthreads();
      if (msg.stop) break;
    }
  }
  __syncthreads();
  for (int i = tid; i < R.nloc; i += kRT) {
    a.x[r0 + i] = sx[i];
    a.vj[r0 + i] = sv[i];
    a.vjm[r0 + i] = svm[i];
    a.wj[r0 + i] = sw[i];
    a.wjm[r0 + i] = swm[i];
  }
  if (blockIdx.x == 0 && tid == 0) {
    a.scal[S_GAM] = gam;
    a.scal[S_GAMP] = gamp;
    a.scal[S_C] = c;
    a.scal[S_CP] = cp;
    a.scal[S_S] = s;
    a.scal[S_SP] = sp;
    a.scal[S_ETA] = eta;
    a.flags[F_ITER] = it;
    a.flags[F_DONE] = done;
    a.flags[F_CONV] = conv;
  }
  if (Group::kCluster) {
    grp.arrive(wid);
    grp.wait(wid);
  }
}

template <class Args>
int run_launch(Ctx* c, SolverData* S, const RunPlan& P, void (*k)(const Args, const RunGroup), const Args& a) {
  RunGroup rg{S->run_slots.p, S->run_bar.p, S->run_halo.p, S->run_neighbours};
  ELFEL_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)P.blocks);
  cfg.blockDim = dim3(kRT);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at[1];
  if (P.cluster) {
    if (P.blocks > 8) ELFEL_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)P.blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    ELFEL_CUDA(c, cudaMemsetAsync(S->run_bar.p, 0, sizeof(unsigned) * kRunWords, c->stream));
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = 1;
  ELFEL_CUDA(c, cudaLaunchKernelEx(&cfg, k, a, rg));
  return ELFEL_OK;
}

template <typename T, bool D16, bool IR>
int cg_launch(Ctx* c, SolverData* S, const RunPlan& P, const CgRun<T>& a) {
  if (P.cluster) return run_launch(c, S, P, cg_run_k<T, D16, IR, true, false, ClusterGroup>, a);
  // FP64: the extra multiply-add per entry pays for the barrier in small systems only
  if (sizeof(T) == 4 || S->nu <= kRunTwoRows64) {
    if (P.ms) return run_launch(c, S, P, cg_run_k<T, D16, IR, true, true, GridGroup>, a);
    return run_launch(c, S, P, cg_run_k<T, D16, IR, false, true, GridGroup>, a);
  }
  if (P.ms) return run_launch(c, S, P, cg_run_k<T, D16, IR, true, false, GridGroup>, a);
  return run_launch(c, S, P, cg_run_k<T, D16, IR, false, false, GridGroup>, a);
}

template <typename T, bool D16>
int mr_launch(Ctx* c, SolverData* S, const RunPlan& P, const MrRun<T>& a) {
  if (P.cluster) return run_launch(c, S, P, mr_run_k<T, D16, true, ClusterGroup>, a);
  if (P.ms) return run_launch(c, S, P, mr_run_k<T, D16, true, GridGroup>, a);
  return run_launch(c, S, P, mr_run_k<T, D16, false, GridGroup>, a);
}

size_t run_smem(int spb, int elem, int vecs, int entries, int d16) {
  return sizeof(double) * kRunPart + (size_t)spb * 32 * elem * vecs + (size_t)spb * sizeof(int2) +
         (size_t)entries * (elem + (d16 ? 2 : 4));
}

}  // namespace

int run_spb_cluster(int64_t nslices) {
  int cl = 1;
  while (cl < 16 && nslices > (int64_t)cl * kRunClusterSlices) cl *= 2;
  return (int)((nslices + cl - 1) / cl);
}

int run_spb_grid(const Ctx* c, int64_t nslices) {
  const int g = std::min(c->sm_count, kRunMaxBlocks);
  return (int)((nslices + g - 1) / g);
}

RunPlan run_plan(Ctx* c, const SolverData* S, int elem, int vecs) {
  RunPlan P;
  const Sell& A = S->A;
  if (!c->one_launch || S->nu < 1 || !S->run_slots.p) return P;
  const int64_t limit = elem == 8 ? kRunClusterRows64 : kRunClusterRows32;
  if (S->nu <= limit) {
    const int spb = run_spb_cluster(A.nslices);
    const size_t sm = run_smem(spb, elem, vecs, S->run_entries[0], A.d16);
    if (sm <= (size_t)kRunSmem) {
      P.spb = spb;
      int cl = 1;
      while ((int64_t)cl * spb < A.nslices) cl *= 2;
      P.blocks = cl;
      P.cluster = P.ms = 1;
      P.max_entries = S->run_entries[0];
      P.smem = sm;
      return P;
    }
  }
  const int spb = run_spb_grid(c, A.nslices);
  const size_t sv = run_smem(spb, elem, vecs, 0, A.d16);
  if (sv > (size_t)kRunSmem) return P;
  const size_t sm = run_smem(spb, elem, vecs, S->run_entries[1], A.d16);
  P.spb = spb;
  P.blocks = (int)((A.nslices + spb - 1) / spb);
  P.ms = sm <= (size_t)kRunSmem ? 1 : 0;
  P.max_entries = S->run_entries[1];
  P.smem = P.ms ? sm : sv;
  return P;
}

int run_cg64(Ctx* c, SolverData* S, const RunPlan& P) {
  const CgRun<double> a{S->view(), S->A.v64.p, S->dinv64.p, S->x64.p, S->r64.p, S->p64.p, S->y64.p, S->z64.p,
                        S->scal.p, S->flags.p, P.spb,       P.max_entries, kRunIters};
  return S->A.d16 ? cg_launch<double, true, false>(c, S, P, a) : cg_launch<double, false, false>(c, S, P, a);
}

int run_cg32(Ctx* c, SolverData* S, const RunPlan& P) {
  const CgRun<float> a{S->view(), S->A.v32.p, S->dinv32.p, S->xa32.p, S->r32.p, S->p32.p, S->zz32.p, S->z32.p,
                       S->scal.p, S->flags.p, P.spb,       P.max_entries, kRunIters};
  return S->A.d16 ? cg_launch<float, true, true>(c, S, P, a) : cg_launch<float, false, true>(c, S, P, a);
}

int run_mr64(Ctx* c, SolverData* S, const RunPlan& P, double* x, double* z, double* vj, double* vjm, double* wj,
             double* wjm) {
  const MrRun<double> a{S->view(), S->A.v64.p, S->dinv64.p, x,     z,             vj,       vjm, wj, wjm,
                        S->scal.p, S->flags.p, P.spb,       P.max_entries, kRunIters};
  return S->A.d16 ? mr_launch<double, true>(c, S, P, a) : mr_launch<double, false>(c, S, P, a);
}

int run_mr32(Ctx* c, SolverData* S, const RunPlan& P, float* x, float* z, float* vj, float* vjm, float* wj,
             float* wjm) {
  const MrRun<float> a{S->view(), S->A.v32.p, S->dinv32.p, x,     z,             vj,       vjm, wj, wjm,
                       S->scal.p, S->flags.p, P.spb,       P.max_entries, kRunIters};
  return S->A.d16 ? mr_launch<float, true>(c, S, P, a) : mr_launch<float, false>(c, S, P, a);
}

}  // namespace elfel
