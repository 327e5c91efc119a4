"""Coefficients read from page-locked host arrays by the integration kernels (HostCoef) against the copied ones (GPU).

The same values by the same kernels: K and F are equal bit for bit, from
aligned and unaligned arrays, and a later call without conductivities uses the ones
given last.
"""
import numpy as np
import pytest
import torch

from problems import elasticity_setup, heat_space

pytestmark = pytest.mark.gpu


def pinned(a, offset):
    """A page-locked copy that starts `offset` doubles into its allocation."""
    t = torch.empty(a.size + offset, dtype=torch.float64).pin_memory()
    v = t.numpy()[offset:]
    v[:] = a.ravel()
    return v.reshape(a.shape), t


def system(E, kind, n):
    if kind == "elasticity":
        mesh, fesp, _, _ = elasticity_setup(E, n, max(1, n // 2))
        return mesh, fesp, {"npts": 3}
    if kind == "T4":
        mesh = E.T4block(1.0, 1.0, 1.0, *(min(n, 20),) * 3)
        fesp = E.FESpace(float, mesh, E.FEH1_T4())
        E.numberdofs(fesp)
        return mesh, fesp, {"npts": 1}
    block = {"Q4": E.Q4block, "Q4x": E.Q4block, "T3": E.T3block}.get(kind, E.T6block)
    fe = {"Q4": E.FEH1_Q4, "Q4x": E.FEH1_Q4, "T3": E.FEH1_T3}.get(kind, E.FEH1_T6)
    mesh = block(1.0, 1.0, n, n)
    if kind == "curved":  # one midside node off its edge
        mesh.xy[mesh.conn[0, 4] - 1] += 0.01 / n
    return mesh, heat_space(E, mesh, fe()), {"kind": "Gauss", "order": 3 if kind == "Q4x" else 2} if kind[0] == "Q" else {"npts": 3}


@pytest.mark.parametrize("kind", ["T6", "curved", "Q4", "Q4x", "T3", "T4", "elasticity"])
@pytest.mark.parametrize("n", [1, 8, 33, 130])
@pytest.mark.parametrize("offset", [0, 1])
def test_same_bits(E, gpu, kind, n, offset):
    mesh, fesp, rule = system(E, kind, n)
    rng = np.random.default_rng(n)
    shape = (mesh.nel, 2) if kind == "elasticity" else (mesh.nel,)
    ndofs = E.ndofs(fesp)
    am = E.start(E.SysmatAssemblerGPU(), ndofs, ndofs)
    qp = E.QPIterator(fesp, rule)
    coef = rng.uniform(0.5, 2.0, shape)

    def assemble(a):
        if kind == "elasticity":
            E.assemble_elasticity(am, E.FEIterator(fesp), qp, 1.0, 0.3, True, a)
        else:
            E.assemble_heat(am, E.FEIterator(fesp), qp, a, -6.0)
        return E.finish(am).data.copy(), am.rhs().copy()

    for _ in range(3):  # records, then bases and tiles
        coef = rng.uniform(0.5, 2.0, shape)
        want = assemble(coef)
        v, keep = pinned(coef, offset)
        got = assemble(v)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        if kind != "elasticity":
            am.heat(None, -6.0)
            assert np.array_equal(E.finish(am).data, want[0])
