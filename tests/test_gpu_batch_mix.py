"""Batches that mix cluster systems and graph systems, and what happens when a step fails (GPU)."""
import numpy as np
import pytest

from problems import heat_space

pytestmark = pytest.mark.gpu


def system(E, ctx, n, seed, etype="T6"):
    """A resident heat system of n x n cells, its start vector and number of unknowns."""
    mesh = E.jitter((E.T6block if etype == "T6" else E.T3block)(1.0, 1.0, n, n), 0.1 / n, seed=seed)
    fesp = heat_space(E, mesh, E.FEH1_T6() if etype == "T6" else E.FEH1_T3())
    nd, nu = E.ndofs(fesp), E.nunknowns(fesp)
    kappa = np.random.default_rng(seed).uniform(0.5, 2.0, mesh.nel)
    am = E.start(E.SysmatAssemblerGPU(ctx=ctx), nd, nd)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), kappa, -6.0)
    T = np.zeros(nd)
    E.gathersysvec(T, fesp)
    return am, T, nu


def run(E, ctx, systems, method, capacity=8, rtol=1e-10):
    b = E.BatchSolver(method, capacity=capacity, ctx=ctx)
    slots = [b.add(am, T, nu, rtol=rtol) for am, T, nu in systems]
    out = b.run(graphs=2)
    b.close()
    return [out[s] for s in slots]


def test_failed_step(E, gpu, monkeypatch):
    """A step fails after its clusters were launched: the graphs of the large system cannot
    be captured on the legacy default stream (an error code, nothing runs).  The batch is
    closed and its memory used again at once; a batch that is kept goes on, with the same bits."""
    monkeypatch.setenv("ELFEL_TUNE", "0")
    ctx = E.Context(0)
    systems = [system(E, ctx, n, n) for n in (30, 20, 12, 104)]
    want = run(E, ctx, systems, "pcg32_ir")
    for keep in (False, True):
        ctx.set_stream(1)  # cudaStreamLegacy
        b = E.BatchSolver("pcg32_ir", capacity=8, ctx=ctx)
        slots = [b.add(am, T, nu, rtol=1e-10) for am, T, nu in systems]
        with pytest.raises(E.ElfelError):
            b.step(50)
        if keep:
            ctx.set_stream(None)
            out = b.run(graphs=2)
            for s, (T, st) in zip(slots, want):
                assert np.array_equal(out[s][0], T) and out[s][1]["iterations"] == st["iterations"]
            b.close()
        else:
            b.close()
            ctx.set_stream(None)
            for (T, st), (T0, st0) in zip(run(E, ctx, systems, "pcg32_ir"), want):
                assert np.array_equal(T, T0) and st["iterations"] == st0["iterations"]


def test_harvest_without_staging(E, gpu, monkeypatch):
    """Without page-locked memory (ELFEL_STAGE=0 stands for none to be had) the finished requests
    of a step are taken one by one: each has its own status, and the same solution."""
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("ELFEL_STAGE", on)
        ctx = E.Context(0)
        srv = E.HeatServer("pcg32_ir", max_active=8, rtol=1e-10, ctx=ctx)
        ids = [srv.submit(E.heat_request(et, n, kappa=k, Q=-3.0, keep_solution=i != 2))
               for i, (et, n, k) in enumerate([("T3", 20, 1.0), ("T6", 12, 1.7), ("T3", 20, 0.6), ("T6", 105, 1.2),
                                               ("T3", 9, 1.3)])]
        res = {r["id"]: r for r in srv.drain()}
        assert sorted(res) == sorted(ids) and all(r["status"] == 0 and r["converged"] for r in res.values())
        out.append([(srv.solution(i), res[i]["iterations"], res[i]["relres"]) for k, i in enumerate(ids) if k != 2])
        with pytest.raises(E.ElfelError):
            srv.solution(ids[2])
        srv.close()
    for (T, it, rr), (T1, it1, rr1) in zip(*out):
        assert np.array_equal(T, T1) and it == it1 and rr == rr1


def test_tuning_is_not_timed_beside_clusters(E, gpu):
    """The grid of the graphs is tuned on the graphs alone: with 20 cluster systems of the largest kind in
    the same step the candidates' times stay within twice those without them (four times, timed beside them)."""
    ms = []
    for crowd in (0, 20):
        ctx = E.Context(0)
        big = system(E, ctx, 130, 1)
        b = E.BatchSolver("pcg32_ir", capacity=64, ctx=ctx)
        others = [system(E, ctx, 98, k) for k in range(crowd)]
        for am, T, nu in [big] + others:
            b.add(am, T, nu, rtol=1e-10)
        b.step(8)
        lines = [line for line, _ in ctx.tuning() if line.startswith("batch_pcg32_ir")]
        assert len(lines) == 1
        ms.append([float(w.split("=")[1].rstrip("*")[:-2]) for w in lines[0].split()[1:]])
        b.run(graphs=2)
        b.close()
    assert min(ms[1]) <= 2.0 * min(ms[0]), ms


def test_many_iterations_in_one_step(E, gpu):
    """A step of 2^26 graphs: 2^32 iterations for a cluster system, more than an int holds; it ends when it has converged."""
    ctx = E.Context(0)
    am, T, nu = system(E, ctx, 6, 1, etype="T3")
    b = E.BatchSolver("pcg32_ir", capacity=2, ctx=ctx)
    s = b.add(am, T, nu, rtol=1e-10)
    assert b.step(1 << 26) == 0 and b.done() == [s]
    assert b.result(s)[1]["converged"]
    b.close()
