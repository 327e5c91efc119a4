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
#include <algorithm>

#include "krylov_dev.cuh"

namespace elfel {

namespace {

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
  const RunRows<T, D16, MS> R(a.A, a.v, (int)blockIdx.x, a.spb, a.max_entries, reinterpret_cast<int2*>(sd + ld));
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
  const RunRows<T, D16, MS> R(a.A, a.v, (int)blockIdx.x, a.spb, a.max_entries, reinterpret_cast<int2*>(swm + ld));
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

}  // namespace

size_t run_smem(int spb, int elem, int vecs, int entries, int d16) {
  return sizeof(double) * kRunPart + (size_t)spb * 32 * elem * vecs + (size_t)spb * sizeof(int2) +
         (size_t)entries * (elem + (d16 ? 2 : 4));
}

int run_spb_cluster(int64_t nslices) {
  int cl = 1;
  while (cl < 16 && nslices > (int64_t)cl * kRunClusterSlices) cl *= 2;
  return (int)((nslices + cl - 1) / cl);
}

int run_spb_grid(const Ctx* c, int64_t nslices) {
  const int g = std::min(c->sm_count, kRunMaxBlocks);
  return (int)((nslices + g - 1) / g);
}

// The smallest power of two of blocks (16 at most) that holds the slices at
// kRunBatchRows rows a block.
int run_spb_batch(int64_t nslices, int elem) {
  const int64_t most = (elem == 4 ? kRunBatchRows32 : kRunBatchRows64) / 32;
  int cl = 1;
  while (cl < 16 && nslices > cl * most) cl *= 2;
  return (int)((nslices + cl - 1) / cl);
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
