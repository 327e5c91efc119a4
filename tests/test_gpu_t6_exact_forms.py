"""The closed-form T6 elasticity and Stokes records (elast_t6_exact_k, stokes_t6_exact_k) against the tabulated kernels (GPU).

A 3-point rule with one weight larger by 6e-14 (relative) is not recognised as
exact and takes the kernels that sum the tabulated reference tensors.  Its
values differ by at most 6e-14 of that point's share of an entry; the share is
at most about twice the largest entry of its block.  Both forms evaluate about
ten sums and products per entry and add up to 8 elements, with terms of a few
times the largest entry: 64 * 2^-53 * 8 = 6e-14.  Together each block of K, F
and the pressure mass stay within 2e-13 of their largest entry.
"""
import numpy as np
import pytest

from problems import elasticity_setup, stokes_setup

pytestmark = pytest.mark.gpu

TOL = 2e-13
SIZES = [(1, 1), (64, 1), (13, 5), (43, 3), (40, 40)]
FORMS = ["square", "sheared", "inverted", "thin", "far"]


def rule(E, fesp, off):
    q = E.QPIterator(fesp, {"npts": 3})
    if off:
        w = np.array(q.quadr.weights, dtype=float).copy()
        w[0] *= 1.0 + 6e-14
        q.quadr.weights = w
    return q


def reshape(xy, form):
    A = {"sheared": [[1.0, 0.3], [0.8, 1.0]], "inverted": [[-1.0, 0.0], [0.2, 1.0]], "thin": [[1.0, 0.0], [0.0, 0.02]]}
    xy = xy @ np.array(A.get(form, np.eye(2)))
    # dyadic offset and coordinates: edge lengths stay exact
    return xy + 8.0 if form == "far" else xy


def close(a, b):
    assert np.abs(a - b).max() <= TOL * np.abs(b).max()


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("plane_strain,load", [(True, True), (False, False)])
def test_elasticity(E, gpu, nx, ny, form, plane_strain, load):
    mesh, fesp, bforce, _ = elasticity_setup(E, nx, ny)
    mesh.xy[:] = reshape(mesh.xy, form)
    n = E.ndofs(fesp)
    out = []
    for off in (False, True):
        am = E.start(E.SysmatAssemblerGPU(), n, n)
        E.assemble_elasticity(am, E.FEIterator(fesp), rule(E, fesp, off), 3.0, 0.3, plane_strain,
                              bforce if load else None)
        out.append((E.finish(am), am.rhs().copy()))
    (K1, F1), (K0, F0) = out
    assert np.array_equal(K1.indptr, K0.indptr) and np.array_equal(K1.indices, K0.indices)
    close(K1.data, K0.data)
    close(F1, F0)


@pytest.mark.parametrize("nx,ny", [(s, s) for s in (1, 3, 8, 9, 41)])
@pytest.mark.parametrize("form", FORMS)
def test_stokes(E, gpu, nx, ny, form):
    vmesh, pmesh, ufesp, pfesp = stokes_setup(E, nx, lid=True)
    vmesh.xy[:] = reshape(vmesh.xy, form)
    n = E.ndofs(ufesp) + E.ndofs(pfesp)
    p = np.zeros(n, dtype=bool)
    p[np.unique(E.FEIterator(pfesp).eldofs_table()) - 1] = True
    out = []
    for off in (False, True):
        am = E.start(E.SysmatAssemblerGPU(), n, n)
        E.assemble_stokes(am, E.FEIterator(ufesp), E.FEIterator(pfesp), rule(E, ufesp, off), 0.7)
        out.append(E.finish(am))
    K1, K0 = out
    assert np.array_equal(K1.indptr, K0.indptr) and np.array_equal(K1.indices, K0.indices)
    cols = np.repeat(np.arange(n), np.diff(K0.indptr))
    mixed = p[cols] | p[K0.indices]
    close(K1.data[~mixed], K0.data[~mixed])
    close(K1.data[mixed], K0.data[mixed])
