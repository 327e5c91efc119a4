// The batched engine's view of a system (batch.cu, batch_run.cu).
#pragma once
#include "solve.cuh"

namespace elfel {

// per-system scalars
enum { B_RZ = 0, B_PQ, B_ALPHA, B_BETA, B_RR, B_RMAX, B_DELTA, B_TOL2, B_BN2, B_SCALE, B_RRT, B_RREC, B_COUNT = 16 };
// per-system ints
enum { I_MODE = 0, I_ITER, I_MAXIT, I_BRK, I_RESTART, I_CONV, I_REPL, I_COUNT = 8 };
enum { M_IDLE = 0, M_CG, M_FOLD, M_RESTART, M_STARTED, M_DONE };

// One system as the batched kernels see it.
struct BSys {
  SellView A;
  const float* v32;
  const double* v64;
  const float* dinv32;
  const double* dinv64;
  const float* rowsum;  // the FP32 matrix's row sums
  float *x32, *r32, *z32, *p32, *q32;
  double *x64, *r64, *z64, *p64, *q64;
  const double* b64;
  int64_t ntiles;
  int sl, pad_;        // row groups of kBlk per tile (1, 4 or 8: fixed per system by its size)
  double* part;        // ntiles x 4 partial sums
  unsigned* ticket;    // work items finished in the current kernel
  const int* nitems;   // work items of this system in the current map
  double* sc;          // B_COUNT scalars
  int* st;             // I_COUNT ints
  int spb, ms, window, room;  // its division in a cluster (batch_run.cu): see RunPlan
  const int4* win;
};

// How a system runs in the batch: in a cluster of `blocks` thread blocks of its
// own (batch_run.cu), or with the others in the graphs (blocks = 0).  A
// function of the system alone, so that its result does not depend on the mix.
struct BRunPlan {
  int blocks = 0, spb = 0, ms = 0, window = 0, room = 0;
  const int4* win = nullptr;
  size_t smem = 0;
};
BRunPlan batch_run_plan(const Ctx* c, const SolverData* S, int ir);
// kBRunIters iterations of each of the n systems list[0..n) (slots of sys,
// device array), one cluster of `blocks` each, on stream st.
constexpr int kBRunIters = 64;
int batch_run_launch(Ctx* c, cudaStream_t st, int ir, const BSys* sys, const int* list, int n, int blocks, size_t smem,
                     int iters);

// One system's FP32 refinement inside one kernel, replacements included
// (elfel_solve): its descriptor, scalars and state on the device.
struct IrOne {
  BSys sys;
  double sc[B_COUNT];
  int st[I_COUNT];
  int list;
};

}  // namespace elfel
