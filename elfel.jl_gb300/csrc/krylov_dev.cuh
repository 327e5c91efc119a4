// Device parts of the one-launch Krylov iterations (krylov.cu, one system;
// batch_run.cu, many): the groups of blocks that iterate together, their
// sums, and a block's part of the matrix.
#pragma once
#include <cooperative_groups.h>

#include "krylov.cuh"

namespace elfel {

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
  __device__ __forceinline__ RunRows(const SellView& A, const T* v, int block, int spb, int max_entries, int2* sbw_sh) {
    const int tid = threadIdx.x;
    const int64_t s0 = (int64_t)block * spb;
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

}  // namespace elfel
