// Device construction of the CSC pattern and of the per-nonzero contributor
// lists (the "slot -> nonzero" map), with the semantics of
// SparseArrays.sparse(I, J, V, m, n) as called by finish! of
// SysmatAssemblerSparse (Elfel.jl src/Assemblers.jl:121-123):
//   * one slot per appended triplet, ordered as the assemble! calls append them;
//   * entries with equal (row, col) are summed in that slot order;
//   * explicitly assembled zeros stay in the pattern;
//   * rows ascend within each column.
//
// Steps (all deterministic; integer atomics only count and bucket):
//   1. column counts (one int32 atomic per column group in block mode, per
//      slot in COO mode)
//   2. exclusive scan -> column starts
//   3. bucket the column groups' numbers (block mode) or each slot's key
//      (row << 32 | slot) (COO mode) into their columns; the order inside a
//      column does not matter, groups and keys carry the slot order
//   4. sort each column's keys in the registers of one thread (merge-exchange
//      networks sized to the longest of the warp's 32 columns; long columns by
//      the whole warp), count its distinct rows, write the storage index of every
//      contribution (contrib) in sorted order and the warp's row starts
//   5. scan -> colptr; copy the row starts to rowval and the first
//      contribution of each nonzero (cptr)
//   6. (at a pattern's second value reduction) the contributor-count order
//      of each window of 128 nonzeros (window_order_k).
#include <type_traits>

#include "pack32.cuh"
#include "sysmat.cuh"

namespace elfel {

constexpr int kWideThreads = 256;  // 8 warps
constexpr int kSortCap = 256;      // keys of a long column sorted in shared memory
constexpr int kColBatch = 32;      // columns of a warp: one per thread

// The sort of a batch of columns by threads, for columns of up to NK keys.
template <int NK>
struct Net {
  static constexpr int kThreads = NK > 48 ? 32 : 128;
  static constexpr int kBlocks = NK > 48 ? 8 : NK == 48 ? 4 : 3;  // an SM
  static constexpr int kGroups = NK > 48 ? 32 : 16;               // column groups of a column (block mode)
  static constexpr int kBatch = NK > 48 ? 3072 : 1240;            // keys of a batch
  static constexpr int kArea = NK > 48 ? 3168 : 1320;             // words of a shared area: kBatch and its padding
  static constexpr int kBits = NK > 64 ? 7 : 6;                   // of a key's place among its column's
  static constexpr uint32_t kSpan = (1u << (32 - kBits)) - 2;     // row span that fits beside it in 32 bits
};
constexpr int kNet = 48;    // block mode, on average at most kNetMean slots a column
constexpr int kNetL = 96;   // block mode, more
// COO mode: 64-bit keys (48 spill).  Triplets with longer columns (plane elasticity on T6, T4)
// go on to sort_wide_k after a look at their lengths.  To CSC with a warp for every column
// (and the values uploaded before the build) and here: T4 36^3 992 and 905 us, elasticity
// 200 x 100 1420 and 1297, T6 200 x 200 807 and 706.
constexpr int kNet64 = 40;
// Slots per column: 16 to 18 on T3, T6 and Q4 meshes (vertices of a T6 mesh 36), 36 in
// plane elasticity on T6 (24 and 72), 48 in Taylor-Hood, 96 on T4.  The larger form keeps
// eight warps an SM instead of 16 and is taken where the other would leave most
// batches to sort_wide_k.  Set-up to CSC with the smaller and the larger form: T6 500 x 500
// 1765 and 2005 us, Q4 700 x 700 1196 and 1287; elasticity 250 x 125 1264 and 1130,
// Taylor-Hood 60 x 60 529 and 455, T4 40^3 920 and 837.
constexpr int kNetMean = 24;

// Block mode: one thread per column group (one atomic per group instead of
// one per slot).  The row tables are the uploaded element DOF tables, range
// checked on upload; the column is checked here.
__global__ void count_groups_k(SlotGen g, int64_t ngroups, int32_t* colcnt, int64_t ncol, int* bad) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < ngroups; q += (int64_t)gridDim.x * blockDim.x) {
    int32_t c;
    int64_t s0;
    int len;
    const int32_t* rt;
    group_info(g, (uint32_t)q, c, s0, len, rt);
    if (c < 0 || c >= ncol) {
      atomicExch(bad, 1);
      continue;
    }
    atomicAdd(&colcnt[c], len);
  }
}

__global__ void count_cols_k(SlotGen g, int64_t n, int32_t* colcnt, int64_t ncol, int64_t nrow, int* bad) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
    int32_t r, c;
    int64_t st;
    slot_rc(g, s, r, c, st);
    if (r < 0 || r >= nrow || c < 0 || c >= ncol) {
      atomicExch(bad, 1);
      continue;
    }
    atomicAdd(&colcnt[c], 1);
  }
}

// Block mode: each group's number into its column, gk[colstart + i] (a column of n
// slots has at most n groups).  A group's rows and slots follow from its number,
// so 4 bytes per group are written and read back instead of 8 per slot
// (500,000 T6 elements: 90 us for the 18M slot keys, 32 us here).
__global__ void bucket_groups_k(SlotGen g, int64_t ngroups, const int64_t* __restrict__ colstart, int64_t ncol,
                                int32_t* cursor, uint32_t* gk) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < ngroups; q += (int64_t)gridDim.x * blockDim.x) {
    int32_t c;
    int64_t s0;
    int len;
    const int32_t* rt;
    group_info(g, (uint32_t)q, c, s0, len, rt);
    if (c < 0 || c >= ncol) continue;
    gk[colstart[c] + atomicAdd(&cursor[c], 1)] = (uint32_t)q;
  }
}

// COO mode.  Consecutive triplets mostly share their column (a local column of
// an element matrix): the lanes of a warp with equal columns in a
// row form a run whose first lane reserves the run's positions with one
// atomic and hands them out by shuffle.
__global__ void bucket_k(SlotGen g, int64_t n, const int64_t* colstart, int64_t nrow, int64_t ncol, int32_t* cursor,
                         uint64_t* keys) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); s0 < n; s0 += stride) {
    const int64_t s = s0 + lane;
    bool valid = s < n;
    int32_t r = 0, c = -1;
    int64_t st;
    if (valid) slot_rc(g, s, r, c, st);
    valid = valid && r >= 0 && r < nrow && c >= 0 && c < ncol;  // as counted
    if (!valid) c = -1;
    const int32_t cprev = __shfl_up_sync(0xffffffffu, c, 1);
    const bool head = lane == 0 || c != cprev;  // lanes without a triplet form runs (c = -1) of their own
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const unsigned upto = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);
    const int start = 31 - __clz(heads & upto);  // first lane of this lane's run
    int32_t base = 0;
    if (head && valid) {
      const unsigned after = heads & ~upto;  // heads of later runs
      const int end = after ? __ffs(after) - 1 : 32;
      base = atomicAdd(&cursor[c], end - lane);
    }
    base = __shfl_sync(0xffffffffu, base, start);
    if (valid) keys[colstart[c] + base + (lane - start)] = ((uint64_t)(uint32_t)r << 32) | (uint64_t)(uint32_t)s;
  }
}

__device__ __forceinline__ void cmpswap(uint64_t* a, int64_t i, int64_t j) {
  uint64_t x = a[i], y = a[j];
  if (x > y) {
    a[i] = y;
    a[j] = x;
  }
}

// Bitonic network in its "flip" form: every comparator puts the smaller key at
// the lower index, so any length n sorts correctly when comparators that reach
// past n are skipped (those positions behave as +infinity).  One warp.  The
// sizes are powers of two below 2^31 (a column holds fewer than 2^31 slots),
// so block and offset come from 32-bit shifts and masks.
__device__ void warp_sort(uint64_t* a, int n, int lane) {
  if (n < 2) return;
  const unsigned un = (unsigned)n;
  int lg = 0;
  while ((1u << lg) < un) ++lg;
  const unsigned half_pairs = 1u << (lg - 1);
  for (int ls = 1; ls <= lg; ++ls) {  // size = 2^ls, h = 2^(ls - 1)
    const int lh = ls - 1;
    const unsigned size = 1u << ls, h = 1u << lh;
    for (unsigned p = lane; p < half_pairs; p += 32) {
      const unsigned blk = p >> lh, off = p & (h - 1);
      const unsigned i = blk * size + off;
      const unsigned j = blk * size + size - 1 - off;
      if (j < un) cmpswap(a, i, j);
    }
    __syncwarp();
    for (int lst = lh - 1; lst >= 0; --lst) {  // stride = 2^lst
      const unsigned stride = 1u << lst;
      for (unsigned p = lane; p < half_pairs; p += 32) {
        const unsigned blk = p >> lst, off = p & (stride - 1);
        const unsigned i = (blk << (lst + 1)) + off;
        const unsigned j = i + stride;
        if (j < un) cmpswap(a, i, j);
      }
      __syncwarp();
    }
  }
}

// Register-resident bitonic sort of P <= 32 keys, one per lane: lanes 0..P-1
// end ascending (every group of P lanes is sorted, in alternating
// directions); shuffles exchange the partners.  Unused lanes hold ~0.
template <int P, typename K>
__device__ __forceinline__ K reg_sort(K v, int lane) {
#pragma unroll
  for (int k = 2; k <= P; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const K o = __shfl_xor_sync(0xffffffffu, v, j);
      const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
      v = keep_min ? (v < o ? v : o) : (v < o ? o : v);
    }
  }
  return v;
}

// Number of keys of a sequence sorted ascending across the warp's lanes
// (one per lane, padding ~0) that are below x (keys are distinct): a binary
// search whose probes are per-lane shuffles.
template <typename K>
__device__ __forceinline__ int count_below(K seq, K x) {
  int pos = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (__shfl_sync(0xffffffffu, seq, pos + step - 1) < x) pos += step;
  if (__shfl_sync(0xffffffffu, seq, pos) < x) ++pos;
  return pos;
}

__device__ __forceinline__ int bit_length(uint32_t x) { return x ? 32 - __clz((int)x) : 0; }

// A column whose row and slot spans fit in 31 bits together is sorted on
// 32-bit packed keys (pack32.cuh): a compare-exchange stage of the register
// sorts then costs half the instructions of the 64-bit one.  The packing of
// the keys of the whole warp (valid keys: lo <= hi per field; lanes without
// keys pass lo = ~0u, hi = 0); false when it does not fit.
__device__ __forceinline__ bool pack_warp(uint32_t rlo, uint32_t rhi, uint32_t slo, uint32_t shi, Pack32* p) {
  const uint32_t rmin = __reduce_min_sync(0xffffffffu, rlo), rmax = __reduce_max_sync(0xffffffffu, rhi);
  const uint32_t smin = __reduce_min_sync(0xffffffffu, slo), smax = __reduce_max_sync(0xffffffffu, shi);
  if (rmax < rmin || smax < smin) return false;
  const int sb = bit_length(smax - smin);
  if (bit_length(rmax - rmin) + sb > 31) return false;
  *p = Pack32{rmin, smin, sb};
  return true;
}

// Output of the sorted columns: each key's storage index goes to contrib[b + t]
// (b = the column's first slot, t = the key's place in it), and the keys that
// start a row (their predecessor has another row) to nzrow / nzpos = (row, b + t):
// in a batch of 32 columns sorted by threads one after the other from the
// batch's first slot, in a batch marked wide[] from each column's first slot.
// compact_k moves them to rowval / cptr once the first nonzeros are known.
struct ColOut {
  int32_t* contrib;
  int32_t* nzrow;
  int32_t* nzpos;
  int32_t* wide;   // of each batch: its columns are sorted by warps
  int32_t* list;   // the batches that are
  int32_t* nlist;  // their number
};

__device__ __forceinline__ void put_key(const SlotGen& g, const ColOut& o, int64_t b, uint64_t key, int t, bool first,
                                        int li) {
  o.contrib[b + t] = (int32_t)slot_store(g, (int64_t)(key & 0xffffffffull));
  if (first) {
    o.nzrow[b + li] = (int32_t)(key >> 32);
    o.nzpos[b + li] = (int32_t)(b + t);
  }
}

// Sort 32 < n <= 64 keys (keys[b + lane], keys[b + 32 + lane]) by merging:
// the first 32 and the other n - 32 are sorted in registers separately, each
// key's place is its index plus the number of keys of the other sequence
// below it; the keys are placed in sh and read back in order.
__device__ __forceinline__ int sort_column_merge(const SlotGen& g, const ColOut& o, int64_t b, int n,
                                                 const uint64_t* keys, uint64_t* sh, int lane) {
  uint64_t v0 = keys[b + lane];
  uint64_t v1 = lane + 32 < n ? keys[b + lane + 32] : ~0ull;
  const int m = n - 32;
  const bool has1 = lane < m;
  const uint32_t r0v = (uint32_t)(v0 >> 32), s0v = (uint32_t)v0;
  const uint32_t r1v = (uint32_t)(v1 >> 32), s1v = (uint32_t)v1;
  Pack32 pk;
  if (pack_warp(has1 ? min(r0v, r1v) : r0v, has1 ? max(r0v, r1v) : r0v, has1 ? min(s0v, s1v) : s0v,
                has1 ? max(s0v, s1v) : s0v, &pk)) {
    uint32_t k0 = pack32(v0, pk), k1 = has1 ? pack32(v1, pk) : ~0u;
    k0 = reg_sort<32>(k0, lane);
    if (m > 16) k1 = reg_sort<32>(k1, lane);
    else if (m > 8) k1 = reg_sort<16>(k1, lane);
    else if (m > 4) k1 = reg_sort<8>(k1, lane);
    else if (m > 1) k1 = reg_sort<4>(k1, lane);
    const int r0 = lane + count_below(k1, k0);
    const int r1 = lane + count_below(k0, k1);
    sh[r0] = unpack32(k0, pk);
    if (has1) sh[r1] = unpack32(k1, pk);
  } else {
    v0 = reg_sort<32>(v0, lane);
    if (m > 16) v1 = reg_sort<32>(v1, lane);
    else if (m > 8) v1 = reg_sort<16>(v1, lane);
    else if (m > 4) v1 = reg_sort<8>(v1, lane);
    else if (m > 1) v1 = reg_sort<4>(v1, lane);
    const int r0 = lane + count_below(v1, v0);
    const int r1 = lane + count_below(v0, v1);
    sh[r0] = v0;
    if (has1) sh[r1] = v1;
  }
  __syncwarp();
  const uint64_t s0 = sh[lane], s1 = lane + 32 < n ? sh[lane + 32] : ~0ull;
  const uint64_t p0 = __shfl_up_sync(0xffffffffu, s0, 1);
  const uint64_t last0 = __shfl_sync(0xffffffffu, s0, 31);
  uint64_t p1 = __shfl_up_sync(0xffffffffu, s1, 1);
  if (lane == 0) p1 = last0;
  const bool f0 = lane == 0 || (s0 >> 32) != (p0 >> 32);
  const bool f1 = lane + 32 < n && (s1 >> 32) != (p1 >> 32);
  const unsigned m0 = __ballot_sync(0xffffffffu, f0), m1 = __ballot_sync(0xffffffffu, f1);
  const unsigned below = (1u << lane) - 1u;
  put_key(g, o, b, s0, lane, f0, __popc(m0 & below));
  if (lane + 32 < n) put_key(g, o, b, s1, lane + 32, f1, __popc(m0) + __popc(m1 & below));
  __syncwarp();  // sh is reused by the warp's next column
  return __popc(m0) + __popc(m1);
}

// Sort one column's keys by (row, slot), write its output (ColOut) and return its
// number of distinct rows (one warp).  Columns of up to 32 keys are sorted in
// registers, up to 64 by sort_column_merge; longer ones with the bitonic
// network in shared memory (up to kSortCap keys, in sh) or in place in global
// memory.
__device__ int sort_column(const SlotGen& g, const ColOut& o, int64_t b, int n, uint64_t* keys,
                           uint64_t* sh, int lane) {
  const unsigned below = (1u << lane) - 1u;
  if (n <= 32) {
    const bool has = lane < n;
    uint64_t v = has ? keys[b + lane] : ~0ull;
    Pack32 pk;
    const uint32_t rv = (uint32_t)(v >> 32), sv = (uint32_t)v;
    if (n > 1 && pack_warp(has ? rv : ~0u, has ? rv : 0u, has ? sv : ~0u, has ? sv : 0u, &pk)) {
      uint32_t k = has ? pack32(v, pk) : ~0u;
      if (n > 16) k = reg_sort<32>(k, lane);
      else if (n > 8) k = reg_sort<16>(k, lane);
      else if (n > 4) k = reg_sort<8>(k, lane);
      else k = reg_sort<4>(k, lane);
      v = has ? unpack32(k, pk) : ~0ull;
    } else {
      if (n > 16) v = reg_sort<32>(v, lane);
      else if (n > 8) v = reg_sort<16>(v, lane);
      else if (n > 4) v = reg_sort<8>(v, lane);
      else if (n > 1) v = reg_sort<4>(v, lane);
    }
    // distinct rows: a key starts a row when its predecessor has another row
    const uint64_t pv = __shfl_up_sync(0xffffffffu, v, 1);
    const bool first = lane < n && (lane == 0 || (v >> 32) != (pv >> 32));
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (lane < n) put_key(g, o, b, v, lane, first, __popc(m & below));
    return __popc(m);
  }
  if (n <= 64) return sort_column_merge(g, o, b, n, keys, sh, lane);
  uint64_t* a;
  if (n <= kSortCap) {
    for (int t = lane; t < n; t += 32) sh[t] = keys[b + t];
    __syncwarp();
    a = sh;
  } else {
    a = keys + b;  // long column: sort in place in global memory
  }
  warp_sort(a, n, lane);
  int32_t cnt = 0;
  for (int t0 = 0; t0 < n; t0 += 32) {
    const int t = t0 + lane;
    bool first = false;
    uint64_t key = 0;
    if (t < n) {
      key = a[t];
      first = (t == 0) || ((key >> 32) != (a[t - 1] >> 32));
    }
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (t < n) put_key(g, o, b, key, t, first, cnt + __popc(m & below));
    cnt += __popc(m);
  }
  __syncwarp();
  return cnt;
}

// Merge exchange (Knuth, The Art of Computer Programming 3, 5.2.2, algorithm M)
// of N keys in registers: the smaller key of every comparator at the lower
// index, so keys of ~0 after the column's own stay behind them.
template <int N, typename K>
__device__ __forceinline__ void net_sort(K (&k)[N]) {
  constexpr int LG = N <= 2 ? 1 : N <= 4 ? 2 : N <= 8 ? 3 : N <= 16 ? 4 : N <= 32 ? 5 : N <= 64 ? 6 : 7;
#pragma unroll
  for (int lp = LG - 1; lp >= 0; --lp) {
    const int p = 1 << lp;
#pragma unroll
    for (int lq = LG - 1; lq >= lp; --lq) {
      const int r = lq == LG - 1 ? 0 : p, d = lq == LG - 1 ? p : (2 << lq) - p;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i + d < N && (i & p) == r) {
          const K x = k[i], y = k[i + d];
          k[i] = min(x, y);
          k[i + d] = max(x, y);
        }
    }
  }
}

// Shared-memory index of word a of a batch: the columns of a warp start n words
// apart, and one word of padding in 32 spreads the usual n (12, 16, 36) over the
// banks.  64-bit keys: one in 16.
__device__ __forceinline__ int pad32(int a) { return a + (a >> 5); }
__device__ __forceinline__ int pad64(int a) { return a + (a >> 4); }

// The batch of columns of a warp, one per lane.
struct Batch {
  int64_t b0;   // first slot
  int total;    // slots
  int off, n;   // of the lane's column: slots before it in the batch, its slots
  int ng;       // its column groups (block mode)
  int nmax, ngmax;
};

// Rows and storage indices of the lane's column, groups in order, to the shared
// areas (T: storage indices, R: rows); returns the column's smallest row and
// whether the row span fits the 32-bit keys.
template <int NG>
__device__ __forceinline__ bool fill_groups(const SlotGen& g, const Batch& B, const uint32_t* gk, int32_t* T, int32_t* R,
                                            uint32_t span, uint32_t* row0) {
  int32_t* Q = T;  // the sorted groups wait at the end of the column's part of T: a group's
                   // entries end at or before its own number, as every later group has one at least
  {
    uint32_t q[NG];
#pragma unroll
    for (int i = 0; i < NG; ++i) q[i] = i < B.ng ? gk[B.b0 + B.off + i] : ~0u;
    net_sort<NG>(q);
#pragma unroll
    for (int i = 0; i < NG; ++i)
      if (i < B.ng) Q[pad32(B.off + B.n - B.ng + i)] = (int32_t)q[i];
  }
  uint32_t lo = ~0u, hi = 0u;
  int p = B.off;
  for (int i = 0; i < B.ng; ++i) {
    const GroupPos G = group_pos(g, (uint32_t)Q[pad32(B.off + B.n - B.ng + i)]);
    const SlotBlock& K = g.b[G.bi];
    const int len = K.transposed ? K.nc : K.nr;
    const int32_t* rt = K.transposed ? K.C + (int64_t)G.e * K.nc : (K.R ? K.R + (int64_t)G.e * K.nr : nullptr);
    const int32_t st = (int32_t)((int64_t)G.e * g.store_per_elem + K.store_off);
    constexpr int U = 6;
    for (int k0 = 0; k0 < len; k0 += U) {
      uint32_t row[U];
#pragma unroll
      for (int u = 0; u < U; ++u) row[u] = rt && k0 + u < len ? (uint32_t)__ldg(rt + k0 + u) : 0u;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u < len) {
          const int k = k0 + u, a = K.transposed ? G.lg : k, b = K.transposed ? k : G.lg;
          T[pad32(p)] = st + (K.sym ? sym_index(a, b) : a + b * K.nr);
          R[pad32(p)] = (int32_t)row[u];
          lo = min(lo, row[u]);
          hi = max(hi, row[u]);
          ++p;
        }
    }
  }
  *row0 = lo;
  return B.ng == 0 || hi - lo <= span;
}

// Row starts of the batch from each lane's sorted rows (row(i), i < n), then
// both shared areas to the output; the batch's contrib has left R.
template <int N, typename F>
__device__ __forceinline__ int put_starts(const ColOut& o, const Batch& B, int lane, int32_t* T, int32_t* R, F row) {
  uint32_t first[(N + 31) / 32] = {};
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < B.n && (i == 0 || row(i) != row(i - 1))) first[i / 32] |= 1u << (i % 32);
  int cnt = 0;
#pragma unroll
  for (int w = 0; w < (N + 31) / 32; ++w) cnt += __popc(first[w]);
  int end = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, end, d);
    if (lane >= d) end += v;
  }
  const int tot = __shfl_sync(0xffffffffu, end, 31);
  int j = end - cnt;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (first[i / 32] >> (i % 32) & 1) {
      T[pad32(j)] = (int32_t)row(i);
      R[pad32(j)] = (int32_t)(B.b0 + B.off + i);
      ++j;
    }
  __syncwarp();
  for (int t = lane; t < tot; t += 32) {
    o.nzrow[B.b0 + t] = T[pad32(t)];
    o.nzpos[B.b0 + t] = R[pad32(t)];
  }
  __syncwarp();  // the areas are reused by the warp's next batch
  return cnt;
}

__device__ __forceinline__ void put_contrib(const ColOut& o, const Batch& B, int lane, const int32_t* R) {
  __syncwarp();
  for (int t = lane; t < B.total; t += 32) o.contrib[B.b0 + t] = R[pad32(t)];
  __syncwarp();
}

// Block mode: keys (row - row0) << BITS | place in slot order.
template <int N, int BITS>
__device__ __forceinline__ int net_groups(const ColOut& o, const Batch& B, int lane, int32_t* T, int32_t* R,
                                          uint32_t row0) {
  uint32_t k[N];
#pragma unroll
  for (int i = 0; i < N; ++i) k[i] = i < B.n ? ((uint32_t)R[pad32(B.off + i)] - row0) << BITS | (uint32_t)i : ~0u;
  net_sort<N>(k);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < B.n) R[pad32(B.off + i)] = T[pad32(B.off + (int)(k[i] & ((1u << BITS) - 1u)))];
  put_contrib(o, B, lane, R);
  return put_starts<N>(o, B, lane, T, R, [&](int i) { return (k[i] >> BITS) + row0; });
}

// COO mode: keys row << 32 | slot, the slot being the storage index.
template <int N>
__device__ __forceinline__ int net_keys(const ColOut& o, const Batch& B, int lane, int32_t* T, int32_t* R,
                                        const uint64_t* keys) {
  uint64_t* K = reinterpret_cast<uint64_t*>(T);  // both areas
  for (int t = lane; t < B.total; t += 32) K[pad64(t)] = keys[B.b0 + t];
  __syncwarp();
  uint64_t k[N];
#pragma unroll
  for (int i = 0; i < N; ++i) k[i] = i < B.n ? K[pad64(B.off + i)] : ~0ull;
  __syncwarp();
  net_sort<N>(k);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < B.n) R[pad32(B.off + i)] = (int32_t)(uint32_t)k[i];
  put_contrib(o, B, lane, R);
  return put_starts<N>(o, B, lane, T, R, [&](int i) { return (uint32_t)(k[i] >> 32); });
}

// The keys of a column of block mode (one warp), for sort_column.
__device__ __forceinline__ void expand_groups(const SlotGen& g, int64_t b, int ng, const uint32_t* gk, uint64_t* keys,
                                              int lane) {
  int64_t at = b;
  for (int i0 = 0; i0 < ng; i0 += 32) {
    int32_t c;
    int64_t s0 = 0;
    int len = 0;
    const int32_t* rt = nullptr;
    if (i0 + lane < ng) group_info(g, gk[b + i0 + lane], c, s0, len, rt);
    int end = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, d);
      if (lane >= d) end += v;
    }
    for (int k = 0; k < len; ++k)
      keys[at + end - len + k] = (uint64_t)(rt ? (uint32_t)rt[k] : 0u) << 32 | (uint64_t)(uint32_t)(s0 + k);
    at += __shfl_sync(0xffffffffu, end, 31);
  }
  __syncwarp();
}

// A warp sorts 32 columns, one per thread, in registers: a network of N keys is
// 2 (32-bit keys) or 6 (64-bit) instructions a comparator and thread, so a column
// of 12 costs about 3 warp instructions and one of 36 about 16 (bitonic sorts across the
// lanes: about 100 and 300).  All global reads and writes of sorted data are
// whole-batch copies through shared memory.  Batches with a longer column,
// more groups, or a row span beyond 26 bits are left to sort_wide_k.
// Measured (500,000 T6 elements, 18M slots): 279 us with one column per warp or
// half warp, 150 us here (60 % of the issue slots idle on instruction fetch of the
// unrolled networks and shared-memory latency at 16 warps an SM).
template <bool COO, int NK>
__global__ void __launch_bounds__(Net<NK>::kThreads, Net<NK>::kBlocks)
    sort_cols_k(SlotGen g, ColOut o, const int64_t* colstart, const int32_t* gcnt, const uint32_t* gk, int64_t ncol,
                const uint64_t* keys, int32_t* nnzcnt) {
  using D = Net<NK>;
  constexpr int W = D::kThreads / 32;
  __shared__ __align__(8) int32_t areas[W][2 * D::kArea];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t *T = areas[wid], *R = areas[wid] + D::kArea;
  const int64_t warps = (int64_t)gridDim.x * W;
  for (int64_t c0 = ((int64_t)blockIdx.x * W + wid) * kColBatch; c0 < ncol;
       c0 += warps * kColBatch) {
    const int64_t c = c0 + lane, c1 = min(c0 + kColBatch, ncol);
    Batch B;
    B.b0 = colstart[c0];
    const int64_t tot = colstart[c1] - B.b0;
    B.off = (int)((c < c1 ? colstart[c] : colstart[c1]) - B.b0);
    B.n = c < c1 ? (int)(colstart[c + 1] - B.b0) - B.off : 0;
    B.ng = !COO && c < c1 ? gcnt[c] : 0;
    B.nmax = __reduce_max_sync(0xffffffffu, B.n);
    B.ngmax = COO ? 0 : __reduce_max_sync(0xffffffffu, B.ng);
    B.total = (int)min(tot, (int64_t)D::kBatch + 1);
    int cnt = 0;
    bool done = false;
    if (B.total <= D::kBatch && B.nmax <= NK && B.ngmax <= D::kGroups) {
      uint32_t row0 = 0;
      bool fit = true;
      if (!COO) {
        if (B.ngmax <= 2) fit = fill_groups<2>(g, B, gk, T, R, D::kSpan, &row0);
        else if (B.ngmax <= 8) fit = fill_groups<8>(g, B, gk, T, R, D::kSpan, &row0);
        else fit = fill_groups<D::kGroups>(g, B, gk, T, R, D::kSpan, &row0);
      }
      if (__all_sync(0xffffffffu, fit)) {
#define NET_COLUMNS(N)                                     \
  do {                                                     \
    if constexpr (COO) cnt = net_keys<N>(o, B, lane, T, R, keys); \
    else cnt = net_groups<N, D::kBits>(o, B, lane, T, R, row0);   \
  } while (0)
        if constexpr (NK <= 48) {
          if (B.nmax <= 6) NET_COLUMNS(6);
          else if (B.nmax <= 12) NET_COLUMNS(12);
          else if (B.nmax <= 18) NET_COLUMNS(18);
          else if (B.nmax <= 24) NET_COLUMNS(24);
          else if (B.nmax <= 36) NET_COLUMNS(36);
          else NET_COLUMNS(NK);
        } else {
          if (B.nmax <= 24) NET_COLUMNS(24);
          else if (B.nmax <= 36) NET_COLUMNS(36);
          else if (B.nmax <= 48) NET_COLUMNS(48);
          else if (B.nmax <= 72) NET_COLUMNS(72);
          else NET_COLUMNS(NK);
        }
#undef NET_COLUMNS
        if (c < c1) nnzcnt[c] = cnt;
        done = true;
      }
    }
    __syncwarp();
    if (lane == 0) {
      const int32_t k = (int32_t)(c0 / kColBatch);
      o.wide[k] = !done;
      if (!done) o.list[atomicAdd(o.nlist, 1)] = k;
    }
  }
}

// The columns of the batches left by sort_cols_k, a warp each: one block per batch.
template <bool COO>
__global__ void __launch_bounds__(kWideThreads) sort_wide_k(SlotGen g, ColOut o, const int64_t* colstart,
                                                           const int32_t* gcnt, const uint32_t* gk, int64_t ncol,
                                                           uint64_t* keys, int32_t* nnzcnt) {
  __shared__ uint64_t sh[kWideThreads / 32][kSortCap];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = *o.nlist;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t k = o.list[i];
    const int64_t c1 = min((k + 1) * kColBatch, ncol);
    for (int64_t c = k * kColBatch + wid; c < c1; c += kWideThreads / 32) {
      const int64_t b = colstart[c];
      if (!COO) expand_groups(g, b, gcnt[c], gk, keys, lane);
      const int cnt = sort_column(g, o, b, (int)(colstart[c + 1] - b), keys, sh[wid], lane);
      if (lane == 0) nnzcnt[c] = cnt;
    }
  }
}

// rowval / cptr from the row starts (ColOut): one warp per batch.
__global__ void compact_k(ColOut o, const int64_t* __restrict__ colstart, const int64_t* __restrict__ colptr,
                          int64_t ncol, int32_t* __restrict__ rowval, int32_t* __restrict__ cptr) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = ((int64_t)gridDim.x * blockDim.x >> 5) * kColBatch;
  for (int64_t c0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kColBatch; c0 < ncol; c0 += stride) {
    const int64_t c1 = min(c0 + kColBatch, ncol);
    const bool wide = o.wide[c0 / kColBatch];
    for (int64_t c = c0; c < c1; c = wide ? c + 1 : c1) {
      const int64_t k0 = colptr[c], cnt = colptr[wide ? c + 1 : c1] - k0, b = colstart[c];
#pragma unroll 4
      for (int64_t i = lane; i < cnt; i += 32) {
        rowval[k0 + i] = o.nzrow[b + i];
        cptr[k0 + i] = o.nzpos[b + i];
      }
    }
  }
}

__global__ void set_last_k(int32_t* cptr, int64_t nnz, int64_t total) { cptr[nnz] = (int32_t)total; }

// For every window of kReduceWindow nonzeros (one warp each): the window's
// nonzeros ordered by contributor count (counts of 8 and more together), ties
// by position -- a stable bucket order; perm[w * kReduceWindow + rank] =
// position in the window.  Positions past the last nonzero sort last.  The
// ranks come from one ballot per bucket and round: rank = items in smaller
// buckets + items of the same bucket in earlier rounds or lower lanes.
constexpr int kOrderBuckets = 8;

__global__ void window_order_k(const int32_t* __restrict__ cptr, int64_t nnz, uint8_t* __restrict__ perm) {
  constexpr int R = kReduceWindow / 32;
  const int lane = threadIdx.x & 31;
  const unsigned lower = (1u << lane) - 1u;
  const int64_t nwin = (nnz + kReduceWindow - 1) / kReduceWindow;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t w = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); w < nwin; w += warps) {
    const int64_t base = w * kReduceWindow;
    const int n = (int)min((int64_t)kReduceWindow, nnz - base);
    int v[R], rank[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = r * 32 + lane;
      v[r] = kOrderBuckets;  // padding: after every bucket
      if (j < n) {
        const int c = cptr[base + j + 1] - cptr[base + j];
        v[r] = (c < 1 ? 1 : (c > kOrderBuckets ? kOrderBuckets : c)) - 1;
      }
      rank[r] = 0;
    }
    int start = 0;
#pragma unroll
    for (int bkt = 0; bkt <= kOrderBuckets; ++bkt) {
      int before = start;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const unsigned m = __ballot_sync(0xffffffffu, v[r] == bkt);
        if (v[r] == bkt) rank[r] = before + __popc(m & lower);
        before += __popc(m);
      }
      start = before;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) perm[base + rank[r]] = (uint8_t)(r * 32 + lane);
  }
}

// Buffers of a build and its steps up to the sorted columns.
struct Build {
  DBuf<int32_t> colcnt, cursor, nzrow, nzpos;
  DBuf<int64_t> colstart;
  DBuf<uint64_t> keys;
  ColOut out;
  int64_t nbatch = 0;
  void release(Ctx* c) {
    colcnt.release(c);
    cursor.release(c);
    nzrow.release(c);
    nzpos.release(c);
    colstart.release(c);
    keys.release(c);
  }
};

static int sort_slots(Ctx* c, const SlotGen& g, int64_t nrow, int64_t ncol, Pattern* P, Build* B) {
  P->release(c);
  const int64_t M = g.total();
  if (M >= (int64_t)0x7fffffff)
    return fail(c, ELFEL_ERR_ARG, "too many assembled entries (%lld): the device pattern holds < 2^31", (long long)M);
  if (nrow >= (int64_t)0x7fffffff || ncol >= (int64_t)0x7fffffff)
    return fail(c, ELFEL_ERR_ARG, "matrix dimension >= 2^31");
  P->nrow = nrow;
  P->ncol = ncol;
  P->nslots = M;
  cudaStream_t st = c->stream;
  // counts, the flag of slots out of range, the number of wide batches, their marks and list (ColOut)
  const int64_t nbatch = B->nbatch = (ncol + kColBatch - 1) / kColBatch;
  ELFEL_TRY(B->colcnt.alloc(c, (size_t)(ncol + 2 + 2 * nbatch)));
  ELFEL_TRY(B->cursor.alloc(c, (size_t)(ncol > 0 ? ncol : 1)));
  ELFEL_TRY(B->colstart.alloc(c, (size_t)ncol + 1));
  int32_t *colcnt = B->colcnt.p, *cursor = B->cursor.p, *bad = colcnt + ncol, *marks = colcnt + ncol + 2;
  int64_t* colstart = B->colstart.p;
  ELFEL_CUDA(c, cudaMemsetAsync(colcnt, 0, sizeof(int32_t) * (ncol + 2), st));
  if (ncol > 0) ELFEL_CUDA(c, cudaMemsetAsync(cursor, 0, sizeof(int32_t) * ncol, st));
  const unsigned gs = grid_for(M, 256, (int64_t)c->sm_count * 16);
  const int64_t ngroups = g.nblocks ? g.nel * (int64_t)g.groups : 0;
  const unsigned gg = grid_for(ngroups, 256, (int64_t)c->sm_count * 16);
  if (M > 0) {
    if (g.nblocks) count_groups_k<<<gg, 256, 0, st>>>(g, ngroups, colcnt, ncol, bad);
    else count_cols_k<<<gs, 256, 0, st>>>(g, M, colcnt, ncol, nrow, bad);
    ELFEL_LAUNCH_CHECK(c);
  }
  ELFEL_TRY(scan_counts_i32(c, colcnt, ncol, colstart));
  const size_t m1 = (size_t)(M > 0 ? M : 1);
  ELFEL_TRY(B->keys.alloc(c, m1));
  // row starts (ColOut), compacted after the scan; the group numbers share the
  // array of the positions (a batch's groups are read before its first row start
  // is written, those of a wide batch's column before the column's)
  ELFEL_TRY(B->nzrow.alloc(c, m1));
  ELFEL_TRY(B->nzpos.alloc(c, m1));
  uint32_t* gk = reinterpret_cast<uint32_t*>(B->nzpos.p);
  uint64_t* keys = B->keys.p;
  if (M > 0) {
    if (g.nblocks) bucket_groups_k<<<gg, 256, 0, st>>>(g, ngroups, colstart, ncol, cursor, gk);
    else bucket_k<<<gs, 256, 0, st>>>(g, M, colstart, nrow, ncol, cursor, keys);
    ELFEL_LAUNCH_CHECK(c);
  }
  // sort + distinct counts (reuse colcnt as per-column nonzero counts)
  ELFEL_TRY(P->contrib.alloc(c, m1));
  const ColOut out = B->out =
      ColOut{P->contrib.p, B->nzrow.p, B->nzpos.p, marks, marks + nbatch, colcnt + ncol + 1};
  if (ncol > 0) {
    const unsigned gwide = grid_for(nbatch, 1, (int64_t)c->sm_count * 8);
    auto sort = [&](auto coo, auto nk) {
      constexpr bool COO = decltype(coo)::value;
      using D = Net<decltype(nk)::value>;
      const unsigned grid = grid_for(nbatch, D::kThreads / 32, (int64_t)c->sm_count * 32);
      sort_cols_k<COO, decltype(nk)::value>
          <<<grid, D::kThreads, 0, st>>>(g, out, colstart, cursor, gk, ncol, keys, colcnt);
      sort_wide_k<COO><<<gwide, kWideThreads, 0, st>>>(g, out, colstart, cursor, gk, ncol, keys, colcnt);
    };
    if (!g.nblocks) sort(std::true_type{}, std::integral_constant<int, kNet64>{});
    else if (M <= kNetMean * ncol) sort(std::false_type{}, std::integral_constant<int, kNet>{});
    else sort(std::false_type{}, std::integral_constant<int, kNetL>{});
    ELFEL_LAUNCH_CHECK(c);
  }
  B->cursor.release(c);
  B->keys.release(c);
  return ELFEL_OK;
}

static int finish_pattern(Ctx* c, int64_t nrow, int64_t ncol, Pattern* P, Build* B) {
  cudaStream_t st = c->stream;
  ELFEL_TRY(P->colptr.alloc(c, (size_t)ncol + 1));
  ELFEL_TRY(scan_counts_i32(c, B->colcnt.p, ncol, P->colptr.p));
  int64_t nnz = 0;
  int hbad = 0;
  ELFEL_TRY(read_back(c, st, {{&nnz, P->colptr.p + ncol, sizeof(nnz)}, {&hbad, B->colcnt.p + ncol, sizeof(hbad)}}));
  if (hbad)  // slots out of range were left out of every step
    return fail(c, ELFEL_ERR_ARG, "assembled row or column number out of range (1..%lld, 1..%lld)", (long long)nrow,
                (long long)ncol);
  P->nnz = nnz;
  ELFEL_TRY(P->rowval.alloc(c, (size_t)(nnz > 0 ? nnz : 1)));
  ELFEL_TRY(P->cptr.alloc(c, (size_t)nnz + 1));
  if (ncol > 0) {
    compact_k<<<grid_for(B->nbatch, 8, (int64_t)c->sm_count * 32), 256, 0, st>>>(B->out, B->colstart.p, P->colptr.p,
                                                                                ncol, P->rowval.p, P->cptr.p);
    ELFEL_LAUNCH_CHECK(c);
  }
  set_last_k<<<1, 1, 0, st>>>(P->cptr.p, nnz, P->nslots);
  ELFEL_LAUNCH_CHECK(c);
  return ELFEL_OK;
}

int build_pattern(Ctx* c, const SlotGen& g0, int64_t nrow, int64_t ncol, Pattern* P) {
  SlotGen g = g0;
  g.prepare();
  Build B;
  int rc = sort_slots(c, g, nrow, ncol, P, &B);
  if (rc == ELFEL_OK) rc = finish_pattern(c, nrow, ncol, P, &B);
  B.release(c);
  if (rc != ELFEL_OK) P->release(c);
  return rc;
}

__global__ void to32_k(int64_t n, const int64_t* a, int32_t* b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (int32_t)a[i];
}

int build_vector_pattern(Ctx* c, const SlotGen& g0, int64_t ncol, Pattern* P) {
  SlotGen g = g0;
  g.prepare();
  Build B;
  auto run = [&]() -> int {
    ELFEL_TRY(sort_slots(c, g, 1, ncol, P, &B));
    ELFEL_TRY(P->cptr.alloc(c, (size_t)ncol + 1));
    to32_k<<<grid_for(ncol + 1, 256, (int64_t)c->sm_count * 16), 256, 0, c->stream>>>(ncol + 1, B.colstart.p, P->cptr.p);
    ELFEL_LAUNCH_CHECK(c);
    return ELFEL_OK;
  };
  const int rc = run();
  B.release(c);
  if (rc != ELFEL_OK) P->release(c);
  return rc;
}

// One thread per nonzero; its contributions are summed left to right, in the
// order the reference's sparse() adds duplicates.
// Each thread reduces kReduceItems nonzeros (k, k + stride, ...) with their
// loads interleaved, so that several independent load chains (cptr ->
// contrib -> record) are in flight per thread; every nonzero still adds its
// contributions in slot order.
constexpr int kReduceItems = 4;

__global__ void reduce_k(const int32_t* __restrict__ cptr, const int32_t* __restrict__ contrib,
                         const double* __restrict__ store, int64_t nnz, double* __restrict__ out) {
  constexpr int R = kReduceItems;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k0 < nnz; k0 += R * stride) {
    int32_t b[R], e[R];
    double s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t k = k0 + i * stride;
      b[i] = 0;
      e[i] = 0;
      if (k < nnz) {
        b[i] = cptr[k];
        e[i] = cptr[k + 1];
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) s[i] = b[i] < e[i] ? store[contrib[b[i]]] : 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (b[i] + 1 < e[i]) s[i] += store[contrib[b[i] + 1]];
#pragma unroll
    for (int i = 0; i < R; ++i)
      for (int32_t t = b[i] + 2; t < e[i]; ++t) s[i] += store[contrib[t]];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t k = k0 + i * stride;
      if (k < nnz) out[k] = s[i];
    }
  }
}

// One warp per window of kReduceWindow nonzeros, four rounds of 32 lanes in
// the window's contributor-count order: the lanes of a round have similar
// counts, so a round issues about as many FP64 adds as its nonzeros need
// (every warp-level FP64 instruction costs the SM's FP64 pipe the same time
// however few of its lanes are active).  Each nonzero still adds its
// contributions in slot order, and the window's values are written inside
// its own 1 KB of the output.
template <bool EARLY = false>
__device__ __forceinline__ void reduce_windows(const int32_t* __restrict__ cptr, const int32_t* __restrict__ contrib,
                                               const uint8_t* __restrict__ perm, const double* store,
                                               int64_t nnz, double* __restrict__ out, unsigned blocks) {
  constexpr int R = kReduceWindow / 32;
  const int lane = threadIdx.x & 31;
  const int64_t nwin = (nnz + kReduceWindow - 1) / kReduceWindow;
  const int64_t warps = (int64_t)blocks * (blockDim.x / 32);
  for (int64_t w = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); w < nwin; w += warps) {
    const int64_t base = w * kReduceWindow;
    const int n = (int)min((int64_t)kReduceWindow, nnz - base);
    int j[R];
    int32_t b[R], e[R];
    double s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      j[r] = perm[base + r * 32 + lane];
      b[r] = 0;
      e[r] = 0;
      if (j[r] < n) {
        b[r] = cptr[base + j[r]];
        e[r] = cptr[base + j[r] + 1];
      }
    }
    if (EARLY) wait_for_previous();
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = b[r] < e[r] ? stored<EARLY>(store + contrib[b[r]]) : 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (b[r] + 1 < e[r]) s[r] += stored<EARLY>(store + contrib[b[r] + 1]);
#pragma unroll
    for (int r = 0; r < R; ++r)
      for (int32_t t = b[r] + 2; t < e[r]; ++t) s[r] += stored<EARLY>(store + contrib[t]);
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (j[r] < n) out[base + j[r]] = s[r];
  }
}

__global__ void __launch_bounds__(256) reduce_win_k(const int32_t* __restrict__ cptr,
                                                   const int32_t* __restrict__ contrib,
                                                   const uint8_t* __restrict__ perm,
                                                   const double* __restrict__ store, int64_t nnz,
                                                   double* __restrict__ out) {
  reduce_windows(cptr, contrib, perm, store, nnz, out, gridDim.x);
}

// The same in the first `blocks` blocks, and a vector's entries (reduce_dense) in
// the others: one launch instead of two for systems whose assembly is mostly
// launches (re-assembly to the host: T3 12 x 12 47.2 -> 43.2 us, T4 4 x 4 x 4 49.8 -> 44.5, plane
// elasticity 20 x 10 50.9 -> 48.1, Taylor-Hood 20 x 20 50.0 -> 45.7).  EARLY: launched
// beside the integration kernel, whose end is waited for after the first window's
// lists are there (T3 12 x 12 43.8 -> 36.2 us, 60 x 60 46.2 -> 38.4; T4, Q4, elasticity and
// Stokes 0 to 2 us less).
template <bool EARLY>
__global__ void __launch_bounds__(256) reduce_win_vec_k(const int32_t* __restrict__ cptr,
                                                       const int32_t* __restrict__ contrib,
                                                       const uint8_t* __restrict__ perm,
                                                       const double* store, int64_t nnz, double* __restrict__ out,
                                                       unsigned blocks, VecRed v) {
  if (blockIdx.x < blocks) {
    reduce_windows<EARLY>(cptr, contrib, perm, store, nnz, out, blocks);
    return;
  }
  if (EARLY) wait_for_previous();
  const int64_t stride = (int64_t)(gridDim.x - blocks) * blockDim.x;
  for (int64_t k = (int64_t)(blockIdx.x - blocks) * blockDim.x + threadIdx.x; k < v.n; k += stride)
    v.out[k] = reduce_entry<EARLY>(v.cptr, v.contrib, v.store, k);
}

// Many reductions in one launch: CTA b serves job k with jobs[k].blk0 <= b <
// jobs[k+1].blk0, items (b - blk0) * blockDim.x onwards.  A dense job
// reduces a vector pattern into the vector (the rhs), else the nnz values.
// Each item adds its contributions in slot order, as reduce_k.
__global__ void reduce_batch_k(const RedJob* __restrict__ jobs, int njobs) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].blk0 <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const RedJob J = jobs[lo];
  const int64_t k = ((int64_t)blockIdx.x - J.blk0) * blockDim.x + threadIdx.x;
  if (k >= J.n) return;
  const int32_t b = J.cptr[k], e = J.cptr[k + 1];
  if (J.dense && b == e) {
    J.out[k] = 0.0;
    return;
  }
  double s = J.store[J.contrib[b]];
  if (J.dense) s = __dadd_rn(0.0, s);  // a vector starts from a zeroed one (SysvecAssembler)
  for (int32_t t = b + 1; t < e; ++t) s += J.store[J.contrib[t]];
  J.out[k] = s;
}

int reduce_batch(Ctx* c, const RedJob* jobs_dev, int njobs, int64_t blocks) {
  if (njobs == 0 || blocks == 0) return ELFEL_OK;
  if (blocks > 0x7fffffff) return fail(c, ELFEL_ERR_ARG, "batched reduction: too many items");
  reduce_batch_k<<<(unsigned)blocks, kRedJobThreads, 0, c->stream>>>(jobs_dev, njobs);
  ELFEL_LAUNCH_CHECK(c);
  return ELFEL_OK;
}

int reduce_values(Ctx* c, Pattern& P, const double* store, double* vals_out, Head* head, VecRed* vec) {
  if (head) head->nnz = 0;
  if (P.nnz == 0) return ELFEL_OK;
  // The count order (window_order_k) pays for itself from a pattern's second
  // reduction on; a pattern reduced once (an end-to-end call) does without it.
  // Both kernels add every nonzero's contributions in slot order: same bits.
  // 1 x n patterns (vectors) are reduced by reduce_dense.
  const bool ordered = P.perm.p != nullptr;  // the order is not being written by the launch before
  if (!P.perm.p && P.reductions >= 1 && P.nrow > 1) {
    const int64_t nwin = (P.nnz + kReduceWindow - 1) / kReduceWindow;
    ELFEL_TRY(P.perm.alloc(c, (size_t)(nwin * kReduceWindow)));
    window_order_k<<<grid_for(nwin, 8, (int64_t)c->sm_count * 16), 256, 0, c->stream>>>(P.cptr.p, P.nnz, P.perm.p);
    ELFEL_LAUNCH_CHECK(c);
  }
  P.reductions++;
  // (a first assembly is followed by a call for the whole CSC, whose indices
  // have the link first, and the auxiliary stream)
  const int64_t hd = head && P.reductions > 1 ? values_head(P.nnz) / kReduceWindow * kReduceWindow : 0;
  auto range = [&](cudaStream_t st, int64_t k0, int64_t n) -> int {  // k0: a multiple of kReduceWindow
    if (P.perm.p) {
      const int64_t nwin = (n + kReduceWindow - 1) / kReduceWindow;
      reduce_win_k<<<grid_for(nwin, 8, (int64_t)c->sm_count * 16), 256, 0, st>>>(
          P.cptr.p + k0, P.contrib.p, P.perm.p + k0, store, n, vals_out + k0);
    } else {
      reduce_k<<<grid_for(n, 256, (int64_t)c->sm_count * 16), 256, 0, st>>>(P.cptr.p + k0, P.contrib.p, store, n,
                                                                            vals_out + k0);
    }
    ELFEL_LAUNCH_CHECK(c);
    return ELFEL_OK;
  };
  if (head) head->nnz = hd;
  if (!hd && P.perm.p && vec && vec->n > 0 && P.nnz < kHeadMinNnz) {
    const int64_t nwin = (P.nnz + kReduceWindow - 1) / kReduceWindow;
    const unsigned gk = grid_for(nwin, 8, (int64_t)c->sm_count * 16);
    const unsigned gv = grid_for(vec->n, 256, (int64_t)c->sm_count * 16);
    const bool early = ordered && P.nnz < kEarlyNnz;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(gk + gv);
    cfg.blockDim = dim3(256);
    cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    ELFEL_CUDA(c, cudaLaunchKernelEx(&cfg, early ? reduce_win_vec_k<true> : reduce_win_vec_k<false>,
                                     (const int32_t*)P.cptr.p, (const int32_t*)P.contrib.p, (const uint8_t*)P.perm.p,
                                     store, P.nnz, vals_out, gk, *vec));
    vec->n = 0;
    return ELFEL_OK;
  }
  if (!hd) return range(c->stream, 0, P.nnz);
  cudaStream_t aux;
  ELFEL_TRY(aux_fork(c, &aux));
  ELFEL_TRY(range(aux, 0, hd));
  ELFEL_CUDA(c, cudaEventRecord(head->ev, aux));
  ELFEL_TRY(range(c->stream, hd, P.nnz - hd));
  ELFEL_CUDA(c, cudaStreamWaitEvent(c->stream, head->ev, 0));
  return ELFEL_OK;
}

__global__ void to_index32_k(const int64_t* src, int64_t n, int64_t limit, int32_t* dst, int* bad) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t v = src[i];
    if (v < 1 || v > limit) {
      atomicExch(bad, 1);
      dst[i] = 0;
    } else {
      dst[i] = (int32_t)(v - 1);
    }
  }
}

// The same conversion reading the (device-readable) host array directly.  Beside
// the pattern build (the auxiliary stream) one block of 64 threads for two SMs, each
// thread with eight 16-byte loads in flight (0.6 MB in all), leaves registers, block
// slots and issue to it; alone on the link, four an SM.  Set-up to CSC of 500,000 T6
// elements: 1698 us; 4 and 1 an SM 1720, 8 and 2 1765, 8 and 8 1814.
constexpr int kHostThreads = 64;

__device__ __forceinline__ int32_t index32(int64_t v, int64_t limit, bool* bad) {
  const bool out = v < 1 || v > limit;
  *bad |= out;
  return out ? 0 : (int32_t)(v - 1);
}

__global__ void __launch_bounds__(kHostThreads) to_index32_host_k(const int64_t* __restrict__ src, int64_t n,
                                                                  int64_t limit, int32_t* __restrict__ dst,
                                                                  int* __restrict__ bad) {
  constexpr int U = 8;
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  bool b = false;
  const int64_t pairs = ((uintptr_t)src & 15) ? 0 : n / 2;  // 16-byte loads where the array allows them
  const longlong2* s2 = reinterpret_cast<const longlong2*>(src);
  int2* d2 = reinterpret_cast<int2*>(dst);
  for (int64_t i0 = tid; i0 < pairs; i0 += U * stride) {
    longlong2 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = i0 + u * stride < pairs ? __ldcs(s2 + i0 + u * stride) : longlong2{1, 1};
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int2 r{index32(v[u].x, limit, &b), index32(v[u].y, limit, &b)};
      if (i0 + u * stride < pairs) d2[i0 + u * stride] = r;
    }
  }
  for (int64_t i0 = 2 * pairs + tid; i0 < n; i0 += U * stride) {
    int64_t v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = i0 + u * stride < n ? __ldcs((const long long*)src + i0 + u * stride) : 1;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int32_t r = index32(v[u], limit, &b);
      if (i0 + u * stride < n) dst[i0 + u * stride] = r;
    }
  }
  if (b) atomicExch(bad, 1);
}

__global__ void copy_host_f64_k(const double* __restrict__ src, int64_t n, double* __restrict__ dst) {
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += U * stride) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = i0 + u * stride < n ? src[i0 + u * stride] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * stride < n) dst[i0 + u * stride] = v[u];
  }
}

int to_index32_direct(Ctx* c, cudaStream_t st, const int64_t* src, int64_t n, int64_t limit, int32_t* dst, int* bad) {
  if (n == 0) return ELFEL_OK;
  const int64_t cap = st == c->stream ? 4 * (int64_t)c->sm_count : (c->sm_count + 1) / 2;
  to_index32_host_k<<<grid_for(n, kHostThreads * 2, cap), kHostThreads, 0, st>>>(src, n, limit, dst, bad);
  ELFEL_LAUNCH_CHECK(c);
  return ELFEL_OK;
}

int copy_host_f64(Ctx* c, cudaStream_t st, const double* src, int pinned, int64_t n, double* dst) {
  if (n == 0) return ELFEL_OK;
  if (pinned) {
    ELFEL_CUDA(c, cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyHostToDevice, st));
    return ELFEL_OK;
  }
  copy_host_f64_k<<<grid_for(n, 256 * 4, (int64_t)c->sm_count * 2), 256, 0, st>>>(src, n, dst);
  ELFEL_LAUNCH_CHECK(c);
  return ELFEL_OK;
}

int to_index32(Ctx* c, const int64_t* src_host, int64_t n, int64_t limit, DBuf<int32_t>* dst, const char* what) {
  ELFEL_TRY(dst->alloc(c, (size_t)(n > 0 ? n : 1)));
  if (n == 0) return ELFEL_OK;
  DBuf<int64_t> tmp;
  DBuf<int> bad;
  ELFEL_TRY(tmp.alloc(c, (size_t)n));
  ELFEL_TRY(bad.alloc(c, 1));
  ELFEL_CUDA(c, cudaMemsetAsync(bad.p, 0, sizeof(int), c->stream));
  ELFEL_CUDA(c, cudaMemcpyAsync(tmp.p, src_host, sizeof(int64_t) * n, cudaMemcpyHostToDevice, c->stream));
  to_index32_k<<<grid_for(n, 256, (int64_t)c->sm_count * 16), 256, 0, c->stream>>>(tmp.p, n, limit, dst->p, bad.p);
  ELFEL_LAUNCH_CHECK(c);
  int hbad = 0;
  ELFEL_CUDA(c, cudaMemcpyAsync(&hbad, bad.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  ELFEL_CUDA(c, cudaStreamSynchronize(c->stream));
  tmp.release(c);
  bad.release(c);
  if (hbad) return fail(c, ELFEL_ERR_ARG, "%s: entry outside 1..%lld", what, (long long)limit);
  return ELFEL_OK;
}

}  // namespace elfel
