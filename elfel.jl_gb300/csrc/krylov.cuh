// One-launch Krylov iterations of one system (krylov.cu).
#pragma once
#include "solve.cuh"

namespace elfel {

constexpr int kRunThreads = 512;
constexpr int kRunMaxBlocks = 160;  // blocks of a grid group (one per SM)
// Cluster groups: slices per block that a cluster is grown for (up to 16
// blocks), and the largest systems that run in one.
constexpr int kRunClusterSlices = 2;
constexpr int64_t kRunClusterRows64 = 16384, kRunClusterRows32 = 32768;
// Beyond this no grid group holds the vectors (226 KB of 20 bytes a row, 160 blocks).
constexpr int64_t kRunGridRows = (int64_t)kRunMaxBlocks * 12000;
constexpr int64_t kRunTwoRows64 = 65536;  // FP64: two barriers an iteration up to here (cg_run_k)
// A batched system takes the smallest cluster whose blocks hold this many rows each.
constexpr int kRunBatchRows32 = 2048, kRunBatchRows64 = 1024;
constexpr int kRunIters = 4096;     // iterations of one launch at most
constexpr int kRunSmem = 227 * 1024 - 1024;  // dynamic shared memory of a block (the kernels' static part apart)

template <bool D16>
struct ColType {
  typedef int16_t type;
};
template <>
struct ColType<false> {
  typedef int32_t type;
};

// A grid group's memory: partial sums [parity][value][block]; words (cleared
// before each launch): arrival counter, error flag, and a flag per block, set
// to the iteration whose rows of the direction are written.  halo: the blocks
// (first, last) that each block gathers from; neighbours: they are at most 32.
constexpr int kRunFlag0 = 32, kRunFlagStride = 8, kRunWords = kRunFlag0 + kRunMaxBlocks * kRunFlagStride;
struct RunGroup {
  double* slots;
  unsigned* words;
  const int2* halo;
  int neighbours;
};

template <typename T>
struct CgRun {
  SellView A;
  const T* v;
  const T* dinv;
  T *x, *r, *p, *p2, *z;  // p2: the second direction buffer
  double* scal;
  int* flags;
  int spb, max_entries, max_iters;
};

template <typename T>
struct MrRun {
  SellView A;
  const T* v;
  const T* minv;
  T *x, *z, *vj, *vjm, *wj, *wjm;
  double* scal;
  int* flags;
  int spb, max_entries, max_iters;
};

// How a system of nslices slices runs: blocks of the group, slices per
// block, cluster or grid, matrix in shared memory.  blocks = 0: not at all
// (too large for the blocks' shared memory).
struct RunPlan {
  int blocks = 0, spb = 0, cluster = 0, ms = 0, max_entries = 0;
  size_t smem = 0;
};

// The slices-per-block values whose largest block entry counts build_sell
// records in SolverData::run_entries: [0] cluster, [1] grid, and of a batched
// system [2] FP32, [3] FP64.
int run_spb_cluster(int64_t nslices);
int run_spb_grid(const Ctx* c, int64_t nslices);
int run_spb_batch(int64_t nslices, int elem);
// Shared memory of a block of spb slices: vecs vectors of elem-byte values
// and, with entries > 0, that many entries of the matrix.
size_t run_smem(int spb, int elem, int vecs, int entries, int d16);
// vecs: vectors of the iteration kept in shared memory (5 for CG, 8 for MINRES).
RunPlan run_plan(Ctx* c, const SolverData* S, int elem, int vecs);

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

}  // namespace elfel
