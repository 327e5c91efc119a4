"""Reductions launched beside the integration kernel (programmatic dependent launch, systems below 2^18 nonzeros) (GPU).

Many re-assemblies with other coefficients each time are issued without waiting
for one another, so that every reduction starts while the records of the call
before are still in memory and new ones are being written.  The values of the
last call are those of a system assembled for the first time with its
coefficients, whose reduction starts after the integration: the same sums in
the same order, equal bit for bit.
"""
import numpy as np
import pytest

from problems import elasticity_setup, heat_space, stokes_setup

pytestmark = pytest.mark.gpu


def systems(E, kind, n):
    """(new system, assemble(system, s)) with coefficients that depend on s."""
    if kind == "elasticity":
        mesh, fesp, bforce, _ = elasticity_setup(E, n, max(1, n // 2))
        qp, it, nd = E.QPIterator(fesp, {"npts": 3}), E.FEIterator(fesp), E.ndofs(fesp)
        first = lambda am, s: E.assemble_elasticity(am, it, qp, 1.0 + s, 0.3, True, s * bforce)  # noqa: E731
        again = lambda am, s: am.elasticity(1.0 + s, 0.3, True, s * bforce)  # noqa: E731
    elif kind == "stokes":
        _, _, ufesp, pfesp = stokes_setup(E, n, lid=True)
        qp, it, pit = E.QPIterator(ufesp, {"npts": 3}), E.FEIterator(ufesp), E.FEIterator(pfesp)
        nd = E.ndofs(ufesp) + E.ndofs(pfesp)
        first = lambda am, s: E.assemble_stokes(am, it, pit, qp, s)  # noqa: E731
        again = lambda am, s: am.stokes(s)  # noqa: E731
    else:
        fe = {"T3": E.FEH1_T3, "T6": E.FEH1_T6, "curved": E.FEH1_T6, "Q4": E.FEH1_Q4, "T4": E.FEH1_T4}[kind]()
        rule = {"kind": "Gauss", "order": 2} if kind == "Q4" else {"npts": 1 if kind == "T4" else 3}
        if kind == "T4":
            mesh = E.T4block(1.0, 1.0, 1.0, n, n, n)
            fesp = E.FESpace(float, mesh, fe)
            E.numberdofs(fesp)
        else:
            mesh = {"T3": E.T3block, "Q4": E.Q4block}.get(kind, E.T6block)(1.0, 1.0, n, n)
            if kind == "curved":
                mesh.xy[mesh.conn[0, 4] - 1] += 0.01 / n
            fesp = heat_space(E, mesh, fe)
        qp, it, nd = E.QPIterator(fesp, rule), E.FEIterator(fesp), E.ndofs(fesp)
        kappa = np.random.default_rng(n).uniform(0.5, 2.0, mesh.nel)
        first = lambda am, s: E.assemble_heat(am, it, qp, s * kappa, -6.0 * s)  # noqa: E731
        again = lambda am, s: am.heat(s * kappa, -6.0 * s)  # noqa: E731
    return (lambda: E.start(E.SysmatAssemblerGPU(), nd, nd)), first, again


@pytest.mark.parametrize("kind,sizes", [("T6", (2, 8, 24, 70)), ("curved", (8, 40)), ("T3", (12, 90)), ("T4", (4, 20)),
                                        ("Q4", (12, 80)), ("elasticity", (8, 40)), ("stokes", (3, 30))])
def test_back_to_back(E, gpu, kind, sizes):
    for n in sizes:
        new, first, again = systems(E, kind, n)
        am = new()
        first(am, 1.0)
        E.finish(am)
        scales = [1.0 + 0.37 * k for k in range(60)]
        for stop in (3, 17, len(scales)):
            for s in scales[:stop]:
                again(am, s)
            K, F = E.finish(am).data.copy(), am.rhs().copy()
            ref = new()
            first(ref, scales[stop - 1])
            assert np.array_equal(K, E.finish(ref).data), (kind, n, stop)
            assert np.array_equal(F, ref.rhs()), (kind, n, stop)
