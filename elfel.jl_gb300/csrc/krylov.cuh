// One-launch Krylov iterations of one system (krylov.cu).
#pragma once
#include "solve.cuh"

namespace elfel {

constexpr int kRunThreads = 512;
constexpr int kRunMaxBlocks = 160;  // blocks of a grid group (one per SM)
// Cluster groups: slices per block that a cluster is grown for (up to 16
// blocks), and the largest systems that run in one (FP64: entries + 8 rows).  Us an
// iteration in a grid and in a cluster, FP64: T6 6,241 unknowns (122,000 by that count) 7.5
// and 6.8, 9,801 (191,000) 7.6 and 8.4; T3 3,481 7.1 and 4.9, 9,801 (147,000) 7.0 and 7.2,
// 22,201 7.2 and 10.3.  FP32: T6 19,321 6.9 and 5.7, 32,041 7.0 and 6.4, from 39,601 on the
// matrix is too large for 16 blocks; T3 32,041 6.9 and 5.9, 47,961 7.0 and 6.7.
constexpr int kRunClusterSlices = 2;
constexpr int64_t kRunClusterWork64 = 180000, kRunClusterRows32 = 32768;
// A batched system takes the smallest cluster whose blocks hold this many rows each.
// Fewer rows a block are faster alone (T6 3,481 unknowns FP32 with 512, 1024, 2048 rows:
// 1.4, 1.5, 1.9 ms), more of them in a crowd (64 of them 14.1, 10.8, 10.0; 64 of 16,129
// 53.6, 53.9, 40.1; a serving burst 12.2, 10.9, 9.3).  FP64 with 512 and 1024: alone 1.9 and
// 2.6 ms, 64 of them 16.1 and 12.3.
constexpr int kRunBatchRows32 = 2048, kRunBatchRows64 = 1024;
// Up to here the windows of the cluster and batch divisions are formed: what 16 blocks can
// hold at the rows above (with the quarter more of batch_run_plan, 40,960) and some room.
constexpr int64_t kRunSmallRows = 65536;
constexpr int kRunIters = 4096;     // iterations of one launch at most
constexpr int kRunSmem = 227 * 1024 - 2048;  // dynamic shared memory of a block (the kernels' static part apart)
constexpr int kRunPart = 3 * kRunThreads + 16;  // doubles of it for the block sums
// The largest system whose vectors the blocks of a grid group hold: a slice of 32 rows takes
// its vectors, the gathered one, and 8 bytes (run_smem without a matrix and a window).
constexpr int64_t run_most_rows(int blocks, int elem, int vecs) {
  return (int64_t)blocks * ((kRunSmem - 8 * kRunPart) / (32 * (vecs + 1) * elem + 8)) * 32;
}
static_assert(run_most_rows(152, 4, 4) == 1634304 && run_most_rows(152, 8, 4) == 822016, "CG, FP32 and FP64");
static_assert(run_most_rows(152, 4, 7) == 1026304 && run_most_rows(152, 8, 7) == 515584, "MINRES, FP32 and FP64");

template <bool D16>
struct ColType {
  typedef int16_t type;
};
template <>
struct ColType<false> {
  typedef int32_t type;
};

// A grid group's memory: partial sums [parity][value][block]; words (cleared
// before each launch): arrival counter, error flag.
struct RunGroup {
  double* slots;
  unsigned* words;
  unsigned spins;  // polls of the arrival counter before a wait gives up
};

// Blocks' column windows in SolverData::run_win: of the cluster division, the
// grid's, and a batched system's (FP32, FP64).
constexpr int kRunWinGrid = 16, kRunWinBatch32 = kRunWinGrid + kRunMaxBlocks, kRunWinBatch64 = kRunWinBatch32 + 16,
              kRunWins = kRunWinBatch64 + 16;

template <typename T>
struct CgRun {
  SellView A;
  const T* v;
  const T* dinv;
  const T* rowsum;  // FP32 (difference form): the row sums
  T *x, *r, *p, *z;
  double* scal;
  int* flags;
  int spb, window, room, max_iters;  // slices, window rows and matrix entries of a block's shared memory
  const int4* win;
  int own_sums;  // FP32: a copy of the row sums in shared memory
};

template <typename T>
struct MrRun {
  SellView A;
  const T* v;
  const T* minv;
  T *x, *z, *vj, *vjm, *wj, *wjm;
  double* scal;
  int* flags;
  int spb, window, room, max_iters;  // slices, window rows and matrix entries of a block's shared memory
  const int4* win;
};

// How a system of nslices slices runs: blocks of the group, slices per
// block, cluster or grid, what lies in shared memory.  blocks = 0: not at all
// (too large for the blocks' shared memory).
struct RunPlan {
  int blocks = 0, spb = 0, cluster = 0, vecs = 0;
  int window = 0;        // rows of the largest column window (0: the direction is gathered from global memory)
  int ms = 0, room = 0;  // matrix in shared memory: entries of the largest block
  size_t smem = 0;
};

// The slices a block takes in each division q of a system: 0 grid, 1 cluster,
// and of a batched system 2 FP32, 3 FP64.  build_sell records the largest
// block's matrix entries (SolverData::run_entries[q]) and the rows of the
// widest column window as one range (run_window[q]) and as two (run_window[4 + q]).
int run_spb_cluster(int64_t nslices);
int run_spb_grid(const Ctx* c, int64_t nslices);
int run_spb_batch(int64_t nslices, int elem);
// Shared memory of a block of spb slices: vecs vectors of elem-byte values, a
// window of that many, and `entries` entries of the matrix.
size_t run_smem(int spb, int elem, int vecs, int window, int entries, int d16);
// vecs: vectors of the iteration kept for a block's own rows (4 for FP64 CG, 5 for FP32 CG, which does with 4 where those do not fit, 7 for MINRES).
// split: the window may be in two ranges (MINRES).
RunPlan run_plan(Ctx* c, const SolverData* S, int elem, int vecs, int least_vecs, int split);

// Up to kRunIters iterations of the FP64 CG, the FP32 CG of the refinement,
// or MINRES in one launch on the context stream; the state is that of the
// graph kernels (S->scal, S->flags, the Krylov vectors), so a paused loop
// goes on with the next call.  MINRES keeps F_ROT: vb/zb/wb are the three-term
// buffers at that rotation.
int run_cg64(Ctx* c, SolverData* S, const RunPlan& P);
int run_cg32(Ctx* c, SolverData* S, const RunPlan& P);
int run_mr64(Ctx* c, SolverData* S, const RunPlan& P, double* x, double* z, double* vj, double* vjm, double* wj,
             double* wjm);
int run_mr32(Ctx* c, SolverData* S, const RunPlan& P, float* x, float* z, float* vj, float* vjm, float* wj,
             float* wjm);

// The FP32 refinement of a system with a window whose matrix and row sums are in
// shared memory, to its end (batch_run.cu): the FP64 residual replacements happen
// inside the kernel, where a host round trip each took 55 us (a solve with
// 12 x 12 T3 elements, 11 replacements: 904 -> 408 us; 64 x 64: 2171 -> 1636; over the
// grid T4 40 x 40 x 40 2762 -> 2279).  A matrix from L2 stays with run_cg32: 808,000 unknowns
// took 90.3 ms here, 88.7 there.  The start is that of run_cg32 (x = 0, r, z, p,
// S_RZ).  Leaves x64, and r64 = b - K x64 of the last replacement.
struct IrResult {
  int iterations, replacements, converged;
};
const int4* run_windows(const SolverData* S, const RunPlan& P);
int run_ir(Ctx* c, SolverData* S, const RunPlan& P, const int4* win, double tol2, double delta, double scale,
                   double bn2, int maxit, IrResult* out);

}  // namespace elfel
