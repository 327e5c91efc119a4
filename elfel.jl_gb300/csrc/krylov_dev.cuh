// Device parts of the one-launch Krylov iterations (krylov.cu, one system;
// batch_run.cu, many): the groups of blocks that iterate together, their
// sums, and a block's part of the matrix.
#pragma once
#include <cooperative_groups.h>

#include "fastdiv64.cuh"
#include "krylov.cuh"

namespace elfel {

namespace cg = cooperative_groups;

constexpr int kRT = kRunThreads;
constexpr int kRW = kRT / 32;

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
      // n is a power of two: only as many steps as there are blocks (an FP64 add
      // and its shuffles take about 100 cycles; a solve with 64 x 64 T3 elements,
      // 16 blocks, 1750 -> 1700 us, 20 x 20, eight, 553 -> 522)
      for (int o = (n < L ? n : L) >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
      for (int k = 0; k < NV; ++k) t[k] = __shfl_sync(0xffffffffu, s, k * L);
    }
    par ^= 1;
  }
  static constexpr bool kCluster = true;
};

struct GridGroup {
  RunGroup g;
  int n, par;
  unsigned target;
  struct Shared {
    int dummy;
  };
  __device__ GridGroup(const RunGroup& rg, Shared*) : g(rg), par(0), target(0) { n = (int)gridDim.x; }
  template <int NV>
  __device__ __forceinline__ void publish(const double (&v)[NV]) {
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) __stcg(g.slots + ((size_t)par * 3 + k) * kRunMaxBlocks + blockIdx.x, v[k]);
    }
  }
  // Thread 0 arrives for the block: a block barrier comes before, so that the
  // release covers the other warps' writes, and one follows wait, so that its
  // acquire covers their reads.  (With a fence on either side instead of the
  // release and acquire forms an iteration took 0.7 us longer: FP64 CG on 129,000
  // unknowns 12.65 -> 11.90 us, FP32 8.62 -> 7.91, on 808,000 15.90 -> 15.25.  Polling
  // by four warps, a separate flag, four counters: 0.8 to 1.9 us longer; pauses
  // between the polls change nothing.)
  __device__ __forceinline__ void arrive(int) {
    target += (unsigned)n;
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.words) : "memory");
    }
  }
  __device__ __forceinline__ bool wait(int wid) {
    if (wid) return true;
    int ok = 1;
    if (threadIdx.x == 0) {
      unsigned spins = 0, v;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.words) : "memory");
        if ((int)(v - target) >= 0) break;
        if (++spins > g.spins || ((spins & 1023u) == 0 && *(volatile unsigned*)(g.words + 1))) {
          atomicExch(g.words + 1, 1u);
          ok = 0;
          break;
        }
      }
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
  }
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
  static constexpr bool kCluster = false;
};

// A thread's part of a dot product.  FP32 terms are added with compensation (Kahan 1965), an
// error of two units of rounding however many rows a thread has (up to 21 at the limit of a
// grid group, five in a batched cluster; the graphs' threads had four rows and one); FP64 plainly.
template <typename T>
struct Dot {
  T s = 0;
  __device__ __forceinline__ void add(T a, T b) { s += a * b; }
};
template <>
struct Dot<float> {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float a, float b) {
    const float y = __fmaf_rn(a, b, -c), t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
};

// The block's sums of the threads' values, in every lane of warp 0 (which
// has room for 3 * kRT doubles in part and 16 in wsum).  FP32 values add
// within the warp in FP32 first; FP64 values go to shared memory as they are.
// nw: the warps that have values (the others' are zero): all, or fewer in a small
// system's block, whose FP64 sums leave the zeros out (run_warps; a solve with 16 x 16 T6
// elements 1119 -> 1076 us, 64 x 64 T3 1700 -> 1644).
template <int NV, typename T>
__device__ __forceinline__ void block_sums(const Dot<T> (&d)[NV], double* part, double* wsum, double (&tot)[NV], int nw) {
  T v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = d[k].s;
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
      // warp w adds the values of warps w, w + 4, ...
      double s = 0.0;
      if (g < NV) {
        const double* p = part + g * kRT + wid * 32 + l;
        if (nw == kRW) {
          s = p[0];
#pragma unroll
          for (int j = 1; j < kRT / 4 / L; ++j) s += p[(j / (32 / L)) * 128 + (j % (32 / L)) * L];
        } else if (wid < nw) {
          s = p[0];
#pragma unroll
          for (int j = 1; j < 32 / L; ++j) s += p[j * L];
          if (wid + 4 < nw) {
#pragma unroll
            for (int j = 0; j < 32 / L; ++j) s += p[128 + j * L];
          }
        }
      }
      quad_total<NV>(lanes_sum<L>(s), wsum, tot);
    }
  }
}

// Warps with values in a block of nsl slices: up to 8 slices go to as many warps
// (RunRows::slice), rows beside one another too.
__device__ __forceinline__ int run_warps(int nsl) { return nsl <= 8 ? nsl : kRW; }

template <typename T>
__device__ __forceinline__ T axpy(T b, T x, T z) {
  return sizeof(T) == 4 ? (T)fmaf((float)b, (float)x, (float)z) : (T)fma((double)b, (double)x, (double)z);
}

// U entries of a row from entry j on: the columns and values of all of them
// are loaded before the gathers, so that U gathers are in flight.  DIFF: each
// term is a_ij (x_j - x_i) (the diagonal slot, which holds the row sum, adds
// nothing: the caller adds it times x_i).
template <typename T, bool D16, bool DIFF, bool MS, int U, typename C, class X>
__device__ __forceinline__ void run_part(const T* v, const C* cols, int row, const X& x, T xi, T (&a)[4]) {
  int cc[U];
  T vv[U], xx[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const C c = MS ? cols[32 * u] : __ldcg(cols + 32 * u);
    cc[u] = D16 ? row + (int)c : (int)c;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) vv[u] = MS ? v[32 * u] : __ldcg(v + 32 * u);
#pragma unroll
  for (int u = 0; u < U; ++u) xx[u] = DIFF ? x[cc[u]] - xi : x[cc[u]];
#pragma unroll
  for (int u = 0; u < U; ++u) a[u & 3] += vv[u] * xx[u];
}

// One row of a slice (its lane's first entry at v, cols; w entries 32 apart),
// the matrix in shared memory (MS) or in global memory.  x is addressed by row
// numbers as they are stored (for a window in shared memory, by its address
// less the window's first row); other blocks rewrite a global x between the
// group's barriers, whose acquire refreshes L1 (plain loads).  X: a pointer,
// or SplitX.  The tail goes in parts of 4, 2 and 1 without predicates: the
// product is bound by instruction issue (and in FP64 a multiply-add left out
// by a predicate costs what it costs).
template <typename T>
struct SplitX {  // the two parts of a window: rows below and from `lo2` on
  const T *a, *b;
  int lo2;
  __device__ __forceinline__ T operator[](int c) const { return (c < lo2 ? a : b)[c]; }
};
template <typename T, bool D16, bool DIFF, bool MS, typename C, class X>
__device__ __forceinline__ T run_row(const T* v, const C* cols, int w, int row, const X& x, T xi) {
  T a[4] = {0, 0, 0, 0};
#define RUN_PART(n)                                           \
  do {                                                        \
    run_part<T, D16, DIFF, MS, n, C, X>(v, cols, row, x, xi, a); \
    v += 32 * n;                                              \
    cols += 32 * n;                                           \
  } while (0)
  for (int j = w >> 3; j > 0; --j) RUN_PART(8);
  if (w & 4) RUN_PART(4);
  if (w & 2) RUN_PART(2);
  if (w & 1) RUN_PART(1);
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
  // sbw_sh: spb slices, followed by `room` entries of the matrix (MS)
  __device__ __forceinline__ RunRows(const SellView& A, const T* v, int block, int spb, int room, int2* sbw_sh) {
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
      C* sc = reinterpret_cast<C*>(sv + room);
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
  // (A x)_i of local row i in slice s; xi: x_i (DIFF: less the row sum times x_i)
  template <bool DIFF, class X>
  __device__ __forceinline__ T row(int s, int i, const X& x, T xi) const {
    const int2 bw = sbw[s];
    const int k = bw.x + (i & 31);
    return run_row<T, D16, DIFF, MS, C, X>(mv + k, mc + k, bw.y, (int)row0 + i, x, xi);
  }
};

// The gathered vector of a block: the rows that its columns lie in (its own
// among them), in shared memory: one range, or two with a gap between them
// (velocity and pressure unknowns).  The block advances all of them itself:
// x = z + beta x (CG) or x = beta z (MINRES), with z of its own rows from
// shared memory and of the others from global memory, where their owners have
// put it before the group's last sum.  The same operations on the same
// operands as the owner's: the same bits.  So only z travels, a product
// gathers from shared memory alone, and the vector needs no barrier of its own.
template <typename T>
struct Window {
  T* x;
  int lo1, n1, lo2, n, own, nown;  // rows [lo1, lo1 + n1), then [lo2, lo2 + n - n1); own rows from x[own] on
  // w: both ranges (see WinArgs in solve.cu); split: keep them apart
  __device__ __forceinline__ Window(T* sh, int4 w, bool split, int row0, int nloc) : x(sh), nown(nloc) {
    lo1 = w.x;
    n1 = (split ? w.y : w.w) - w.x;
    lo2 = split ? w.z : w.w;
    n = n1 + w.w - lo2;
    own = row0 < lo1 + n1 ? row0 - lo1 : n1 + row0 - lo2;
    if (nloc == 0) n = n1 = own = 0;
  }
  __device__ __forceinline__ const T* by_row() const { return x - lo1; }
  __device__ __forceinline__ SplitX<T> by_row_split() const { return SplitX<T>{x - lo1, x + n1 - lo2, lo2}; }
  __device__ __forceinline__ int row(int j) const { return j < n1 ? lo1 + j : lo2 + (j - n1); }
  __device__ __forceinline__ void load(const T* g) {
    for (int j = threadIdx.x; j < n; j += kRT) x[j] = g[row(j)];
  }
  // mine: z of the own rows; g: z of all rows; CG: x = z + beta x, else x = beta z
  template <bool CG>
  __device__ __forceinline__ void advance(const T* mine, const T* g, T beta) {
    const int nh = n - nown;  // rows of others: x[0, own) and x[own + nown, n)
    constexpr int U = 4;
    for (int h0 = threadIdx.x; h0 < nh; h0 += U * kRT) {
      T zz[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int h = h0 + u * kRT, j = h < own ? h : h + nown;
        if (h < nh) zz[u] = g[row(j)];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int h = h0 + u * kRT, j = h < own ? h : h + nown;
        if (h < nh) x[j] = CG ? axpy<T>(beta, x[j], zz[u]) : zz[u] * beta;
      }
    }
    for (int i = threadIdx.x; i < nown; i += kRT)
      x[own + i] = CG ? axpy<T>(beta, x[own + i], mine[i]) : mine[i] * beta;
  }
};

}  // namespace elfel
