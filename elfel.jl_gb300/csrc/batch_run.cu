// Small systems of a batch, each iterated by a thread-block cluster of its own:
// the CG loop of krylov.cu with the whole state machine of the batched engine
// (batch.cu) inside the kernel, kBRunIters iterations a launch.
//
// What bounds it.  In the graphs of three kernels an iteration of a batch of
// small systems cost 21 us, the latency of three kernels, however little work
// it held.  A cluster needs no grid-wide barrier: its systems' blocks meet at
// the hardware cluster barrier (0.2-0.3 us), and the clusters of a launch run
// side by side and independently.  A system takes 1 to 16 blocks by its size
// alone, at most 2048 rows a block in FP32 (the vectors, 41 KB, and the
// matrix, about 140 KB for quadratic triangles, fit a block's shared memory),
// so that a burst of requests spreads over the SMs, and its sums do not depend
// on the mix: the same bits alone, in any mix and whenever it joins.
#include <type_traits>

#include "batch.cuh"
#include "krylov_dev.cuh"

namespace elfel {

namespace {

// One sum over the group (all threads; the totals, and whether the wait ended, are valid in warp 0).
template <int NV, typename T, class Group>
__device__ __forceinline__ bool group_sum(Group& grp, const Dot<T> (&v)[NV], double* part, double* wsum, double (&t)[NV],
                                          int nw = kRW) {
  const int wid = threadIdx.x >> 5;
  block_sums<NV>(v, part, wsum, t, nw);
  if (wid == 0) grp.publish(t);
  grp.arrive(wid);
  const bool ok = grp.wait(wid);
  grp.collect(wid, wsum, t);
  return ok;
}

// A grid group's wait is warp 0's: the block learns here that it ended (false: it ran out).
template <class Group>
__device__ __forceinline__ bool group_done(bool ok, RunMsg& msg) {
  if (Group::kCluster) return true;
  if (threadIdx.x == 0) msg.stop = ok ? M_CG : M_DONE;
  __syncthreads();
  return msg.stop == M_CG;
}

template <bool IR, bool D16, bool MS, class Group>
__device__ __forceinline__ void batch_run(const BSys& S, Group& grp, int rank, uint8_t* smem, RunMsg& msg, int iters) {
  typedef typename std::conditional<IR, float, double>::type T;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  double* part = reinterpret_cast<double*>(smem);
  double* wsum = part + 3 * kRT;
  T* sx = reinterpret_cast<T*>(part + kRunPart);
  const int ld = S.spb * 32;
  T *sr = sx + ld, *sq = sr + ld, *sd = sq + ld, *ss = sd + ld, *pw = ss + (IR ? ld : 0);
  T* const gx = IR ? (T*)S.x32 : (T*)S.x64;
  T* const gr = IR ? (T*)S.r32 : (T*)S.r64;
  T* const gp = IR ? (T*)S.p32 : (T*)S.p64;
  const T* const gd = IR ? (const T*)S.dinv32 : (const T*)S.dinv64;
  T* const gz = IR ? (T*)S.z32 : (T*)S.z64;
  const RunRows<T, D16, MS> R(S.A, IR ? (const T*)S.v32 : (const T*)S.v64, rank, S.spb, S.room,
                              reinterpret_cast<int2*>(pw + S.window));
  const int64_t r0 = R.row0;
  const int nw = run_warps(R.nsl);
  Window<T> W(pw, S.win[rank], false, (int)r0, R.nloc);
  T* const sp = pw + W.own;
  W.load(gp);
  for (int i = tid; i < R.nloc; i += kRT) {
    sx[i] = gx[r0 + i];
    sr[i] = gr[r0 + i];
    sd[i] = gd[r0 + i];
    if (IR) ss[i] = (T)S.rowsum[r0 + i];
  }
  // the system's scalars (warp 0 uses them)
  const double scale = S.sc[B_SCALE], tol = S.sc[B_TOL2], bn2 = S.sc[B_BN2];
  const double thr = IR ? tol : tol * bn2, delta2 = S.sc[B_DELTA] * S.sc[B_DELTA];
  double rz = S.sc[B_RZ], rr = S.sc[B_RR], rmax2 = S.sc[B_RMAX] * S.sc[B_RMAX], pq = 0.0;
  double inv_rz = 0.0, low2 = delta2 * rmax2;
  int it = S.st[I_ITER], brk = S.st[I_BRK], repl = S.st[I_REPL], conv = 0, mode = M_CG;
  const int maxit = S.st[I_MAXIT];
  __syncthreads();

  T be = 0;
  bool keep = true;  // the window holds the direction already
  for (int k = 0; k < iters; ++k) {
    if (!keep) {  // p = z + beta p
      W.template advance<true>(sq, gz, be);
      __syncthreads();
    }
    keep = false;
    // q = A p; p.q (and r.p) -> alpha
    constexpr int N1 = IR ? 2 : 1;
    Dot<T> d1[N1];
    for (int n = 0; n * kRW < R.nsl; ++n) {
      const int s = R.slice(wid, n);
      const int i = s * 32 + lane;
      if (i < R.nloc) {
        const T pi = sp[i];
        T acc = R.template row<IR>(s, i, W.by_row(), pi);
        if (IR) acc += ss[i] * pi;
        sq[i] = acc;
        d1[0].add(acc, pi);
        if (IR) d1[N1 - 1].add(sr[i], pi);
      }
    }
    double t1[N1];
    bool ok = group_sum<N1>(grp, d1, part, wsum, t1, nw);
    if (wid == 0) {
      pq = t1[0];
      const double alpha = pos_finite(pq) ? fast_div(IR ? t1[N1 - 1] : rz, pq) : 0.0;
      if (lane == 0) {
        msg.c[0] = alpha;
        if (!Group::kCluster) msg.stop = ok ? M_CG : M_DONE;
      }
    }
    __syncthreads();
    if (!Group::kCluster && msg.stop == M_DONE) {
      mode = M_DONE;
      break;
    }
    // r -= alpha q, z = D r (kept in q); r.z, r.r (and z.r_old) -> beta
    constexpr int N2 = IR ? 3 : 2;
    const T al = (T)msg.c[0];
    Dot<T> d2[N2];
    for (int i = tid; i < R.nloc; i += kRT) {
      const T ro = sr[i];
      const T ri = ro - al * sq[i];
      sr[i] = ri;
      const T zi = sd[i] * ri;
      sq[i] = zi;
      gz[r0 + i] = zi;
      d2[0].add(ri, zi);
      d2[1].add(ri, ri);
      if (IR) d2[N2 - 1].add(zi, ro);
    }
    double t2[N2];
    block_sums<N2>(d2, part, wsum, t2, nw);
    if (wid == 0) grp.publish(t2);
    grp.arrive(wid);
    for (int i = tid; i < R.nloc; i += kRT) sx[i] += al * sp[i];
    if (wid == 0) inv_rz = IR ? fast_rcp(rz) : rcp_ahead(rz);
    ok = grp.wait(wid);
    grp.collect(wid, wsum, t2);
    if (wid == 0) {
      // (FP32: r.z is 0 or a normal double)
      const double beta = IR ? (t2[0] - t2[N2 - 1]) * inv_rz : times_rcp(t2[0], rz, inv_rz);
      rz = t2[0];
      rr = t2[1];
      ++it;
      conv = le_pos(rr, thr);
      const bool bad = !pos_finite(pq) || !finite(rz) || !finite(rr);
      if (IR) {
        if (bad) {
          brk = 1;
          mode = M_FOLD;
        } else {
          if (lt_pos(rmax2, rr)) {
            rmax2 = rr;
            low2 = delta2 * rmax2;
          }
          if (conv) brk = 2;  // spent directions: restart from p = z
          if (conv || it >= maxit || lt_pos(rr, low2)) mode = M_FOLD;
        }
      } else if (conv && !bad && it < maxit) {
        mode = M_FOLD;  // the recurrence says converged: check the true residual
      } else if (conv || bad || it >= maxit) {
        conv = conv && !bad;
        mode = M_DONE;
      }
      if (!ok) {
        conv = 0;
        mode = M_DONE;
      }
      if (lane == 0) {
        msg.c[0] = beta;
        msg.stop = mode;
      }
    }
    __syncthreads();
    mode = msg.stop;
    if (mode == M_DONE) break;
    be = (T)msg.c[0];
    if (mode == M_FOLD) {
      // the next direction, x64 += s x32 (FP32), then the true residual
      // b - K x64 in FP64
      for (int i = tid; i < R.nloc; i += kRT) {
        sp[i] = axpy<T>(be, sp[i], sq[i]);
        if (IR) {
          S.x64[r0 + i] += scale * (double)sx[i];
          sx[i] = 0;
        } else {
          S.x64[r0 + i] = (double)sx[i];
        }
      }
      if (!Group::kCluster) __syncthreads();
      grp.arrive(wid);
      ok = grp.wait(wid);
      if (!group_done<Group>(ok, msg)) {
        mode = M_DONE;
        break;
      }
      Dot<double> d[1];
      for (int s = wid; s < R.nsl; s += kRW) {
        const int i = s * 32 + lane;
        const double acc = sell_row_resid<D16, true>(S.A, S.v64, S.x64, r0 / 32 + s, lane);
        if (i < R.nloc) {
          const double rv = S.b64[r0 + i] - acc;
          S.r64[r0 + i] = rv;
          d[0].add(rv, rv);
        }
      }
      double t[1];
      ok = group_sum<1>(grp, d, part, wsum, t);
      if (wid == 0) {
        const double rrt = t[0];
        ++repl;
        conv = (!(rrt > 0.0) && finite(rrt)) || rrt <= tol * bn2;
        conv = conv && ok;
        if (conv || !ok || !finite(rrt) || it >= maxit || (!IR && repl > 50)) {
          mode = M_DONE;
        } else {
          // FP32: keep the direction unless the recurrence broke down or its
          // residual drifted far below the true one; FP64: restart
          const double rrec = rr * scale * scale;
          const int restart = !IR || brk || !(rrec > 0.0) || !(rrec >= 1e-6 * rrt);
          brk = 0;
          mode = restart ? M_RESTART : M_STARTED;
          rmax2 = IR ? rrt / (scale * scale) : rmax2;
          low2 = delta2 * rmax2;
        }
        if (lane == 0) {
          msg.c[0] = rrt;
          msg.stop = mode;
        }
      }
      __syncthreads();
      mode = msg.stop;
      if (mode == M_DONE) break;
      const double inv = 1.0 / scale;
      Dot<T> dz[1];
      for (int s = wid; s < R.nsl; s += kRW) {
        const int i = s * 32 + lane;
        if (i < R.nloc) {
          const T ri = IR ? (T)(S.r64[r0 + i] * inv) : (T)S.r64[r0 + i];
          sr[i] = ri;
          const T zi = sd[i] * ri;
          gp[r0 + i] = mode == M_RESTART ? zi : sp[i];
          dz[0].add(ri, zi);
        }
      }
      double t3[1];
      ok = group_sum<1>(grp, dz, part, wsum, t3);
      if (wid == 0) rz = t3[0];
      if (!group_done<Group>(ok, msg)) {
        mode = M_DONE;
        break;
      }
      mode = M_CG;
      W.load(gp);  // the sum's barrier has made it visible
      keep = true;
      __syncthreads();
    }
  }
  __syncthreads();
  for (int i = tid; i < R.nloc; i += kRT) {
    gx[r0 + i] = sx[i];
    gr[r0 + i] = sr[i];
    if (mode == M_CG) gp[r0 + i] = keep ? sp[i] : axpy<T>(be, sp[i], sq[i]);
  }
  if (rank == 0 && tid == 0) {
    S.sc[B_RZ] = rz;
    S.sc[B_RR] = rr;
    S.sc[B_PQ] = pq;
    S.sc[B_RMAX] = sqrt(rmax2);
    S.st[I_ITER] = it;
    S.st[I_BRK] = brk;
    S.st[I_REPL] = repl;
    S.st[I_CONV] = conv;
    S.st[I_MODE] = mode;
  }
}

template <bool IR>
__global__ void __launch_bounds__(kRT, 1) batch_run_k(const BSys* __restrict__ sys, const int* __restrict__ list,
                                                     int iters) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ ClusterGroup::Shared gsh;
  __shared__ RunMsg msg;
  __shared__ BSys S;
  ClusterGroup grp(RunGroup(), &gsh);
  static_assert(sizeof(BSys) % 8 == 0 && sizeof(BSys) / 8 <= kRT, "descriptor staging");
  if (threadIdx.x < sizeof(BSys) / 8)
    reinterpret_cast<uint64_t*>(&S)[threadIdx.x] =
        reinterpret_cast<const uint64_t*>(sys + list[blockIdx.x / grp.n])[threadIdx.x];
  __syncthreads();
  if (S.st[I_MODE] == M_CG) {
    if (S.A.d16) {
      if (S.ms) batch_run<IR, true, true>(S, grp, grp.rank, smem, msg, iters);
      else batch_run<IR, true, false>(S, grp, grp.rank, smem, msg, iters);
    } else {
      if (S.ms) batch_run<IR, false, true>(S, grp, grp.rank, smem, msg, iters);
      else batch_run<IR, false, false>(S, grp, grp.rank, smem, msg, iters);
    }
  }
  grp.arrive(0);  // no block leaves while another may still write its shared memory
  grp.wait(0);
}

}  // namespace

BRunPlan batch_run_plan(const Ctx* c, const SolverData* S, int ir) {
  BRunPlan P;
  if (!c->one_launch || S->nu < 1) return P;
  const int elem = ir ? 4 : 8;
  const int spb = run_spb_batch(S->A.nslices, elem);
  const int entries = S->run_entries[ir ? 2 : 3];
  const int window = S->run_window[ir ? 2 : 3] + (S->run_window[ir ? 2 : 3] & 1);
  if (window == 0) return P;  // too large for the division
  const size_t sv = run_smem(spb, elem, ir ? 5 : 4, window, 0, S->A.d16);
  const size_t sm = run_smem(spb, elem, ir ? 5 : 4, window, entries, S->A.d16);
  // a system whose matrix does not fit iterates from L2 as long as its rows
  // are few (a quarter more than 16 full blocks); larger ones are left to the graphs, which
  // use the whole device.  Ms in the cluster and in graphs, one system and 16: FP32 T6 38,025
  // unknowns 7.3 and 17.1, 24.1 and 62.0; 47,961 (beyond) 8.8 and 20.4, 29.0 and 78.6.  FP64 18,769
  // 6.8 and 11.9, 22.8 and 32.6; 25,281 (beyond) 10.6 and 13.7, 32.6 and 46.0; 62,001 30.8 and
  // 24.4, 90.8 and 117.  So the line could lie further out.
  if (sv > (size_t)kRunSmem || spb * 32 > (ir ? kRunBatchRows32 : kRunBatchRows64) * 5 / 4) return P;
  P.ms = sm <= (size_t)kRunSmem;
  P.spb = spb;
  P.blocks = 1;
  while ((int64_t)P.blocks * spb < S->A.nslices) P.blocks *= 2;
  P.room = P.ms ? entries : 0;
  P.window = window;
  P.win = S->run_win.p + (ir ? kRunWinBatch32 : kRunWinBatch64);
  P.smem = P.ms ? sm : sv;
  return P;
}

int batch_run_launch(Ctx* c, cudaStream_t st, int ir, const BSys* sys, const int* list, int n, int blocks, size_t smem,
                     int iters) {
  auto k = ir ? batch_run_k<true> : batch_run_k<false>;
  ELFEL_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kRunSmem));
  if (blocks > 8) ELFEL_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(n * blocks));
  cfg.blockDim = dim3(kRT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)blocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  ELFEL_CUDA(c, cudaLaunchKernelEx(&cfg, k, sys, list, iters));
  return ELFEL_OK;
}

// One system's refinement over the whole grid (matrix in shared memory).
template <bool D16>
__global__ void __launch_bounds__(kRT, 1) ir_grid_k(const IrOne* __restrict__ one, RunGroup rg, int iters) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ GridGroup::Shared gsh;
  __shared__ RunMsg msg;
  __shared__ BSys S;
  GridGroup grp(rg, &gsh);
  if (threadIdx.x < sizeof(BSys) / 8)
    reinterpret_cast<uint64_t*>(&S)[threadIdx.x] = reinterpret_cast<const uint64_t*>(&one->sys)[threadIdx.x];
  __syncthreads();
  batch_run<true, D16, true>(S, grp, (int)blockIdx.x, smem, msg, iters);
}

static int ir_grid_launch(Ctx* c, SolverData* S, const RunPlan& P, const IrOne* one) {
  auto k = S->A.d16 ? ir_grid_k<true> : ir_grid_k<false>;
  ELFEL_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P.smem));
  ELFEL_CUDA(c, cudaMemsetAsync(S->run_bar.p, 0, 2 * sizeof(unsigned), c->stream));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)P.blocks);
  cfg.blockDim = dim3(kRT);
  cfg.dynamicSmemBytes = P.smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const RunGroup rg{S->run_slots.p, S->run_bar.p, c->run_spins};
  ELFEL_CUDA(c, cudaLaunchKernelEx(&cfg, k, one, rg, (int)kRunIters));
  return ELFEL_OK;
}

// The descriptor and the start of one system's refinement (run_ir).
__global__ void ir_start_k(IrOne* one, BSys d, const double* scal, double tol2, double delta, double scale, double bn2,
                           int maxit) {
  const int t = threadIdx.x;
  if (t < B_COUNT)
    one->sc[t] = t == B_RZ      ? scal[S_RZ]
                 : t == B_TOL2  ? tol2
                 : t == B_DELTA ? delta
                 : t == B_SCALE ? scale
                 : t == B_BN2   ? bn2
                 : t == B_RMAX  ? 1.0
                                : 0.0;
  if (t < I_COUNT) one->st[t] = t == I_MAXIT ? maxit : t == I_MODE ? M_CG : 0;
  if (t == 0) {
    d.sc = one->sc;
    d.st = one->st;
    one->sys = d;
    one->list = 0;
  }
}

int run_ir(Ctx* c, SolverData* S, const RunPlan& P, const int4* win, double tol2, double delta, double scale,
                   double bn2, int maxit, IrResult* out) {
  if (!S->ir_one.p) ELFEL_TRY(S->ir_one.alloc(c, sizeof(IrOne)));
  IrOne* one = reinterpret_cast<IrOne*>(S->ir_one.p);
  BSys d;
  memset(&d, 0, sizeof(d));
  d.A = S->view();
  d.v32 = S->A.v32.p;
  d.v64 = S->A.v64.p;
  d.dinv32 = S->dinv32.p;
  d.dinv64 = S->dinv64.p;
  d.rowsum = S->rowsum32.p;
  d.x32 = S->xa32.p;
  d.r32 = S->r32.p;
  d.z32 = S->z32.p;
  d.p32 = S->p32.p;
  d.x64 = S->x64.p;
  d.r64 = S->r64.p;
  d.b64 = S->b64.p;
  d.spb = P.spb;
  d.ms = P.ms;
  d.window = P.window;
  d.room = P.room;
  d.win = win;
  ir_start_k<<<1, 32, 0, c->stream>>>(one, d, S->scal.p, tol2, delta, scale, bn2, maxit);
  ELFEL_LAUNCH_CHECK(c);
  int st[I_COUNT];
  do {
    unsigned bar[2] = {0, 0};
    if (P.cluster) {
      ELFEL_TRY(batch_run_launch(c, c->stream, 1, &one->sys, &one->list, 1, P.blocks, P.smem, kRunIters));
      ELFEL_TRY(read_back(c, c->stream, {{st, one->st, sizeof(st)}}));
    } else {
      ELFEL_TRY(ir_grid_launch(c, S, P, one));
      ELFEL_TRY(read_back(c, c->stream, {{st, one->st, sizeof(st)}, {bar, S->run_bar.p, sizeof(bar)}}));
    }
    if (bar[1]) return fail(c, ELFEL_ERR_TIMEOUT, "solve: a barrier of the iteration kernel timed out");
  } while (st[I_MODE] == M_CG);
  out->iterations = st[I_ITER];
  out->replacements = st[I_REPL];
  out->converged = st[I_CONV];
  return ELFEL_OK;
}

}  // namespace elfel
