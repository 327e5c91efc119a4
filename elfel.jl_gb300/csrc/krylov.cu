// One-launch Krylov iterations: the CG loop of one system inside a single
// kernel, the row slices of the SELL matrix divided over the thread blocks of
// a group that stays resident for the whole loop.
//
// What bounds it.  As a graph of three kernels an iteration of a system that
// fits the L2 cost 21 us at 961 unknowns and 26 us at 129k: every kernel
// waited for its flags and scalars, re-read the vectors of its rows, and ended
// in a last-block reduction, each a chain of memory round trips and of FP64
// adds (64 cycles apiece).  Here
//   - a thread block keeps the same rows for the whole solve: x, r, q and the
//     preconditioner stay in shared memory, the matrix too when it fits (MS),
//     and the gathered direction of all rows that the block's columns touch
//     (Window), which the block advances itself: only z of the rows around its
//     own travels between blocks;
//   - the sums go thread -> warp -> block -> group, and one warp of every
//     block forms alpha, beta and the convergence test from the group totals
//     (the same partials in the same order: the same bits in every block);
//   - x is advanced between the arrival at and the wait for the second sum.
// Per iteration, quadratic heat, FP64 and FP32 (graphs, then one launch):
//       961 unknowns  21.3 ->  5.4 us   25.8 ->  4.7 us
//     14161           21.1 ->  7.7      21.9 ->  5.6
//    128881           26.2 -> 12.0      22.2 ->  7.8
//    358801           40.2 -> 22.6      32.0 -> 11.2
//    808201           62.7 -> 47.2      45.9 -> 15.8
// MINRES (Taylor-Hood cavity) 27.2 -> 11.1 us at 9026 unknowns.  What is left
// at 128881: the two sums over the grid (1.5 us a barrier with the blocks' uneven
// arrival, 0.8 to collect), in FP64 the FP64 unit (4.5 us), in FP32 at 808201 the
// compensated sums (0.1; 0.3 when a row is added at once).  Measured and not kept: the direction gathered
// from global memory after a barrier of its own (FP32 9.4 us at 128881, 21.1 at
// 808201: gathers that miss L1), 1024 threads a block (17.5 at 808201), the
// next chunk of the matrix prefetched into registers (no change), the matrix
// streamed through rings in shared memory with cp.async (19.0 at 808201), columns and
// FP32 values in quads for 16-byte loads (15.6; 12.4 at 128881 in FP64).
// Two groups are provided:
//   ClusterGroup  one cluster of up to 16 blocks: sums through distributed
//                 shared memory, the hardware cluster barrier (0.2-0.3 us);
//   GridGroup     one block per SM, launched cooperatively: an arrival counter
//                 in global memory (1.1 to 1.25 us a barrier of 152 blocks by
//                 itself).  Every wait is bounded; a wait that runs out marks the
//                 error word and ends the kernel, and the solve starts again in
//                 graphs (or_in_graphs in solve.cu).
#include <algorithm>

#include "krylov_dev.cuh"

namespace elfel {

namespace {

// CG on the permuted system.  IR: the FP32 recurrence of the refinement
// (difference form, flexible step, Polak-Ribiere beta; stops for a residual
// replacement), else FP64 Jacobi PCG.  The recurrences and stopping rules are
// those of the graph kernels (sell_cg_spmv_k, cg_update_k, cg_p_k).
//
// WIN: the direction of the block's column window lies in shared memory
// (Window), two sums an iteration.  Otherwise (columns from everywhere) it is
// gathered from global memory, where a third barrier completes it.
template <typename T, bool D16, bool IR, bool MS, bool WIN, class Group>
__global__ void __launch_bounds__(kRT, 1) cg_run_k(const CgRun<T> a, const RunGroup rg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ typename Group::Shared gsh;
  __shared__ RunMsg msg;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  double* part = reinterpret_cast<double*>(smem);
  double* wsum = part + 3 * kRT;
  T* sx = reinterpret_cast<T*>(part + kRunPart);
  const int ld = a.spb * 32;
  T *sr = sx + ld, *sq = sr + ld, *sd = sq + ld, *ss = sd + ld, *pw = ss + (a.own_sums ? ld : 0);
  const RunRows<T, D16, MS> R(a.A, a.v, (int)blockIdx.x, a.spb, a.room, reinterpret_cast<int2*>(pw + a.window));
  const int r1 = (int)R.row0 + R.nloc, nw = run_warps(R.nsl);
  Window<T> W(pw, WIN ? a.win[blockIdx.x] : make_int4((int)R.row0, r1, r1, r1), false, (int)R.row0, R.nloc);
  T* const sp = pw + W.own;
  W.load(a.p);
  for (int i = tid; i < R.nloc; i += kRT) {
    sx[i] = a.x[R.row0 + i];
    sr[i] = a.r[R.row0 + i];
    sd[i] = a.dinv[R.row0 + i];
    if (IR && a.own_sums) ss[i] = a.rowsum[R.row0 + i];
  }
  const T* const rs = IR && !a.own_sums ? a.rowsum + R.row0 : ss;  // row sums: of the own rows, or where they are
  // the loop's scalars (warp 0 uses them)
  double rz = a.scal[S_RZ], rr = a.scal[S_RR], pq = 0.0, alpha = 0.0, beta = 0.0, inv_rz = 0.0;
  const double thr = a.scal[S_TOL2] * (IR ? a.scal[S_BN2S] : a.scal[S_BN2]);
  const double delta2 = IR ? a.scal[S_DELTA] * a.scal[S_DELTA] : 0.0;
  double rmax2 = a.scal[S_RMAX] * a.scal[S_RMAX];  // the largest r.r since the last replacement
  double low2 = delta2 * rmax2;
  int it = a.flags[F_ITER], done = 0, conv = 0, ru = 0, brk = a.flags[F_BRK];
  const int maxit = a.flags[F_MAXIT];
  Group grp(rg, &gsh);
  __syncthreads();

  T be = 0;
  for (int k = 0; k < a.max_iters; ++k) {
    if (k > 0) {  // p = z + beta p
      if (WIN) {
        W.template advance<true>(sq, a.z, be);
        __syncthreads();
      } else {
        for (int i = tid; i < R.nloc; i += kRT) {
          const T pn = axpy<T>(be, sp[i], sq[i]);
          sp[i] = pn;
          a.p[R.row0 + i] = pn;
        }
        // the new direction is complete before the gathers
        if (!Group::kCluster) __syncthreads();
        grp.arrive(wid);
        const bool ok = grp.wait(wid);
        if (!Group::kCluster) {
          if (tid == 0) msg.stop = ok ? 0 : 2;
          __syncthreads();
          if (msg.stop) break;
        }
      }
    }
    // q = A p; p.q (and r.p) -> alpha
    constexpr int N1 = IR ? 2 : 1;
    Dot<T> d1[N1];
    T la = 0, lp = 0, lr = 0;
    for (int n = 0; n * kRW < R.nsl; ++n) {
      const int s = R.slice(wid, n);
      const int i = s * 32 + lane;
      if (i < R.nloc) {
        const T pi = sp[i];
        if (IR) {  // the row before, while this one's entries are on their way
          d1[0].add(la, lp);
          d1[N1 - 1].add(lr, lp);
        }
        T acc = R.template row<IR>(s, i, WIN ? W.by_row() : (const T*)a.p, pi);
        if (IR) acc += rs[i] * pi;
        sq[i] = acc;
        if (IR) {
          la = acc;
          lp = pi;
          lr = sr[i];
        } else {
          d1[0].add(acc, pi);
        }
      }
    }
    if (IR) {
      d1[0].add(la, lp);
      d1[N1 - 1].add(lr, lp);
    }
    double t1[N1];
    block_sums<N1>(d1, part, wsum, t1, nw);
    if (wid == 0) grp.publish(t1);
    grp.arrive(wid);
    bool ok = grp.wait(wid);
    grp.collect(wid, wsum, t1);
    if (wid == 0) {
      pq = t1[0];
      alpha = pos_finite(pq) ? fast_div(IR ? t1[N1 - 1] : rz, pq) : 0.0;
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
    Dot<T> d2[N2];
    for (int i = tid; i < R.nloc; i += kRT) {
      const T ro = sr[i];
      const T ri = ro - al * sq[i];
      sr[i] = ri;
      const T zi = sd[i] * ri;
      sq[i] = zi;
      if (WIN) a.z[R.row0 + i] = zi;
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
      const double rzn = t2[0];
      rr = t2[1];
      // (FP32: r.z is 0 or a normal double)
      beta = IR ? (rzn - t2[N2 - 1]) * inv_rz : times_rcp(rzn, rz, inv_rz);
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
    be = (T)msg.c[0];
    if (msg.stop) break;
  }
  __syncthreads();
  for (int i = tid; i < R.nloc; i += kRT) {
    a.x[R.row0 + i] = sx[i];
    a.r[R.row0 + i] = sr[i];
    a.p[R.row0 + i] = axpy<T>(be, sp[i], sq[i]);  // the recurrence's next direction
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
// divisions) runs in warp 0 with the divisions side by side in its lanes.
// WIN: the normalised z of the block's column window is in shared memory, and
// what travels is z' before its normalisation, written ahead of the sum that
// gives its norm; otherwise z is gathered from global memory after a barrier.
template <typename T, bool D16, bool MS, bool WIN, class Group>
__global__ void __launch_bounds__(kRT, 1) mr_run_k(const MrRun<T> a, const RunGroup rg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ typename Group::Shared gsh;
  __shared__ RunMsg msg;
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  double* part = reinterpret_cast<double*>(smem);
  double* wsum = part + 3 * kRT;
  T* sx = reinterpret_cast<T*>(part + kRunPart);
  const int ld = a.spb * 32;
  T *sq = sx + ld, *sm = sq + ld, *sv = sm + ld, *svm = sv + ld, *sw = svm + ld, *swm = sw + ld, *zw = swm + ld;
  const RunRows<T, D16, MS> R(a.A, a.v, (int)blockIdx.x, a.spb, a.room, reinterpret_cast<int2*>(zw + a.window));
  const int64_t r0 = R.row0;
  const int r1 = (int)r0 + R.nloc, nw = run_warps(R.nsl);
  Window<T> W(zw, WIN ? a.win[blockIdx.x] : make_int4((int)r0, r1, r1, r1), true, (int)r0, R.nloc);
  T* const sz = zw + W.own;
  W.load(a.z);
  for (int i = tid; i < R.nloc; i += kRT) {
    sx[i] = a.x[r0 + i];
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

  T zs = 0;
  bool moved = false;  // sq holds the next z, not normalised yet
  for (int k = 0; k < a.max_iters && !done; ++k) {
    if (k > 0) {  // z = z' / gamn
      moved = false;
      if (WIN) {
        W.template advance<false>(sq, a.z, zs);
        __syncthreads();
      } else {
        for (int i = tid; i < R.nloc; i += kRT) {
          const T zn = sq[i] * zs;
          sz[i] = zn;
          a.z[r0 + i] = zn;
        }
        if (!Group::kCluster) __syncthreads();
        grp.arrive(wid);
        const bool ok = grp.wait(wid);
        if (!Group::kCluster) {
          if (tid == 0) msg.stop = ok ? 0 : 2;
          __syncthreads();
          if (msg.stop) break;
        }
      }
    }
    // q = A z, delta = q.z
    Dot<T> d1[1];
    for (int n = 0; n * kRW < R.nsl; ++n) {
      const int sl = R.slice(wid, n);
      const int i = sl * 32 + lane;
      if (i < R.nloc) {
        const T zi = sz[i];
        const T acc = WIN ? R.template row<false>(sl, i, W.by_row_split(), zi)
                          : R.template row<false>(sl, i, (const T*)a.z, zi);
        sq[i] = acc;
        d1[0].add(acc, zi);
      }
    }
    double t[1];
    block_sums<1>(d1, part, wsum, t, nw);
    if (wid == 0) grp.publish(t);
    grp.arrive(wid);
    bool ok = grp.wait(wid);
    grp.collect(wid, wsum, t);
    double delta = 0.0;
    if (wid == 0) {
      delta = t[0];
      const double ca = fast_div(delta, gam);
      if (lane == 0) {
        msg.c[0] = ca;
        msg.c[1] = bcoef;
        msg.stop = ok ? 0 : 2;
      }
    }
    __syncthreads();
    if (msg.stop) break;
    // v' = q - (delta/gam) v_j - (gam/gamp) v_{j-1}, z' = M v' (in q), gamn^2 = z'.v'
    const T ca = (T)msg.c[0], cb = (T)msg.c[1];
    Dot<T> d2[1];
    for (int i = tid; i < R.nloc; i += kRT) {
      const T vv = sq[i] - ca * sv[i] - cb * svm[i];
      svm[i] = vv;
      const T zz = sm[i] * vv;
      sq[i] = zz;
      if (WIN) a.z[r0 + i] = zz;
      d2[0].add(zz, vv);
    }
    block_sums<1>(d2, part, wsum, t, nw);
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
    done = stop;
    zs = (T)msg.c[0];
    moved = true;
    const T ca3 = (T)msg.c[1], ca2 = (T)msg.c[2], cia = (T)msg.c[3], cce = (T)msg.c[4];
    // w' = (z - a3 w_{j-1} - a2 w_j) / a1, x += c eta w'
    for (int i = tid; i < R.nloc; i += kRT) {
      const T w = (sz[i] - ca3 * swm[i] - ca2 * sw[i]) * cia;
      swm[i] = w;
      sx[i] += cce * w;
    }
    T* tv = sv;
    sv = svm;
    svm = tv;
    T* tw = sw;
    sw = swm;
    swm = tw;
  }
  __syncthreads();
  for (int i = tid; i < R.nloc; i += kRT) {
    a.x[r0 + i] = sx[i];
    if (moved) a.z[r0 + i] = sq[i] * zs;
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
  RunGroup rg{S->run_slots.p, S->run_bar.p, c->run_spins};
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
    ELFEL_CUDA(c, cudaMemsetAsync(S->run_bar.p, 0, 2 * sizeof(unsigned), c->stream));
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
  if (P.cluster && P.window) return run_launch(c, S, P, cg_run_k<T, D16, IR, true, true, ClusterGroup>, a);
  if (P.cluster) return run_launch(c, S, P, cg_run_k<T, D16, IR, true, false, ClusterGroup>, a);
  if (P.window && P.ms) return run_launch(c, S, P, cg_run_k<T, D16, IR, true, true, GridGroup>, a);
  if (P.window) return run_launch(c, S, P, cg_run_k<T, D16, IR, false, true, GridGroup>, a);
  return run_launch(c, S, P, cg_run_k<T, D16, IR, false, false, GridGroup>, a);
}

template <typename T, bool D16>
int mr_launch(Ctx* c, SolverData* S, const RunPlan& P, const MrRun<T>& a) {
  if (P.cluster && P.window) return run_launch(c, S, P, mr_run_k<T, D16, true, true, ClusterGroup>, a);
  if (P.cluster) return run_launch(c, S, P, mr_run_k<T, D16, true, false, ClusterGroup>, a);
  if (P.window && P.ms) return run_launch(c, S, P, mr_run_k<T, D16, true, true, GridGroup>, a);
  if (P.window) return run_launch(c, S, P, mr_run_k<T, D16, false, true, GridGroup>, a);
  return run_launch(c, S, P, mr_run_k<T, D16, false, false, GridGroup>, a);
}

}  // namespace

size_t run_smem(int spb, int elem, int vecs, int window, int entries, int d16) {
  return sizeof(double) * kRunPart + ((size_t)spb * 32 * vecs + window) * elem + (size_t)spb * sizeof(int2) +
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

RunPlan run_plan(Ctx* c, const SolverData* S, int elem, int vecs, int least_vecs, int split) {
  const Sell& A = S->A;
  if (!c->one_launch || S->graphs || S->nu < 1 || !S->run_slots.p) return RunPlan();
  // A cluster saves about 5000 cycles an iteration at its barriers and sums; in
  // FP64 its 16 SMs take half a cycle over 16 per multiply-add (entries, and
  // about 8 per row for the vectors), which makes that up at 180k of them.
  const bool small = elem == 8 ? A.nnz_pad + 8 * S->nu <= kRunClusterWork64 : S->nu <= kRunClusterRows32;
  for (int cluster = small ? 1 : 0; cluster >= 0; --cluster) {
    RunPlan P;
    const int q = cluster ? 1 : 0;
    P.cluster = cluster;
    P.spb = cluster ? run_spb_cluster(A.nslices) : run_spb_grid(c, A.nslices);
    P.blocks = 1;
    if (cluster)
      while ((int64_t)P.blocks * P.spb < A.nslices) P.blocks *= 2;
    else
      P.blocks = (int)((A.nslices + P.spb - 1) / P.spb);
    // Every row of a window that is not the block's own costs a multiply-add a
    // product (FP64: half a cycle of the SM), which pays for the barrier that
    // the window saves up to these widths.  Us an iteration with the window and without,
    // by the rows beyond the own ones: FP64 cluster 1163 (T4 20^3) 7.5 and 7.6, 2468 (cavity
    // 20 x 20) 8.6 and 8.5; FP64 grid 3519 (T4 40^3) 10.4 and 10.8, 6597 (56^3) 17.2 and 17.0,
    // 9851 (70^3) 24.4 and 23.7; FP32 cluster 2468 6.2 and 6.9, 6447 (cavity 32 x 32) 8.7 and
    // 8.6; FP32 grid 9851 23.8 and 26.3, 16426 (T4 90^3) 28.2 and 32.7, 23472 (cavity 128 x
    // 128) 15.8 and 14.1.
    const int wide = S->run_window[split ? 4 + q : q];
    const int most = P.spb * 32 + (cluster ? 2000 : 8000) * (elem == 8 ? 1 : 2);
    P.window = wide > 0 && wide <= most ? wide + (wide & 1) : 0;  // even: 8-byte alignment of what follows
    auto smem = [&](int entries) {
      return run_smem(P.spb, elem, P.vecs, P.window ? P.window : P.spb * 32, entries, A.d16);
    };
    P.vecs = vecs;
    if (smem(0) > (size_t)kRunSmem) P.vecs = std::min(vecs, least_vecs);
    if (smem(0) > (size_t)kRunSmem) P.window = 0;
    const size_t sv = smem(0), sm = smem(S->run_entries[q]);
    P.ms = sm <= (size_t)kRunSmem;
    if (cluster && !P.ms) continue;  // a grid has room
    if (!P.ms && sv > (size_t)kRunSmem) return RunPlan();
    if (!P.window) P.ms = cluster;  // (the grid's form without a window reads the matrix from L2)
    P.room = P.ms ? S->run_entries[q] : 0;
    P.smem = P.ms ? sm : sv;
    return P;
  }
  return RunPlan();
}

// The window argument of a launch: the room for it (without one, for the own
// rows of the direction), and the blocks' windows.
static int run_window_arg(const RunPlan& P) { return P.window ? P.window : P.spb * 32; }
const int4* run_windows(const SolverData* S, const RunPlan& P) { return S->run_win.p + (P.cluster ? 0 : kRunWinGrid); }

int run_cg64(Ctx* c, SolverData* S, const RunPlan& P) {
  const CgRun<double> a{S->view(), S->A.v64.p, S->dinv64.p, nullptr, S->x64.p, S->r64.p, S->p64.p, S->z64.p,
                        S->scal.p, S->flags.p, P.spb, run_window_arg(P), P.room, kRunIters, run_windows(S, P), P.vecs > 4};
  return S->A.d16 ? cg_launch<double, true, false>(c, S, P, a) : cg_launch<double, false, false>(c, S, P, a);
}

int run_cg32(Ctx* c, SolverData* S, const RunPlan& P) {
  const CgRun<float> a{S->view(), S->A.v32.p, S->dinv32.p, S->rowsum32.p, S->xa32.p, S->r32.p, S->p32.p, S->z32.p,
                       S->scal.p, S->flags.p, P.spb, run_window_arg(P), P.room, kRunIters, run_windows(S, P), P.vecs > 4};
  return S->A.d16 ? cg_launch<float, true, true>(c, S, P, a) : cg_launch<float, false, true>(c, S, P, a);
}

int run_mr64(Ctx* c, SolverData* S, const RunPlan& P, double* x, double* z, double* vj, double* vjm, double* wj,
             double* wjm) {
  const MrRun<double> a{S->view(), S->A.v64.p, S->dinv64.p, x,     z,             vj,       vjm, wj, wjm,
                        S->scal.p, S->flags.p, P.spb, run_window_arg(P), P.room, kRunIters, run_windows(S, P)};
  return S->A.d16 ? mr_launch<double, true>(c, S, P, a) : mr_launch<double, false>(c, S, P, a);
}

int run_mr32(Ctx* c, SolverData* S, const RunPlan& P, float* x, float* z, float* vj, float* vjm, float* wj,
             float* wjm) {
  const MrRun<float> a{S->view(), S->A.v32.p, S->dinv32.p, x,     z,             vj,       vjm, wj, wjm,
                       S->scal.p, S->flags.p, P.spb, run_window_arg(P), P.room, kRunIters, run_windows(S, P)};
  return S->A.d16 ? mr_launch<float, true>(c, S, P, a) : mr_launch<float, false>(c, S, P, a);
}

}  // namespace elfel
