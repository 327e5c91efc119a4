"""The tensor-product form of the 2 x 2 Gauss rule on Q4 elements (heat_q4_gauss2_k) against the per-point kernel (GPU).

A rule whose last weight is one ulp larger is not recognised as the 2 x 2 rule
and takes the per-point kernel; its values differ by an ulp of that point's
share.  Tolerance: both forms evaluate the same sums of about 40 products per
entry, whose terms do not exceed a few times the element's largest entry:
K within 40 * 2^-53 * 8 = 4e-14 of the largest entry of K, the same for F.
"""
import numpy as np
import pytest

from problems import heat_space

pytestmark = pytest.mark.gpu

TOL = 4e-14


def both(E, mesh, order, kappa, Q=-6.0):
    fesp = heat_space(E, mesh, E.FEH1_Q4())
    n = E.ndofs(fesp)
    out = []
    for off in (False, True):
        q = E.QPIterator(fesp, {"kind": "Gauss", "order": 2})
        q.quadr.param_coords = q.quadr.param_coords[order]
        w = np.array(q.quadr.weights, dtype=float).copy()
        if off:
            w[3] = np.nextafter(w[3], 2.0)
        q.quadr.weights = w
        am = E.start(E.SysmatAssemblerGPU(), n, n)
        E.assemble_heat(am, E.FEIterator(fesp), q, kappa, Q)
        out.append((E.finish(am), am.rhs().copy()))
    return out


@pytest.mark.parametrize("nx,ny", [(1, 1), (127, 1), (64, 2), (43, 3), (300, 5)])
@pytest.mark.parametrize("order", [[0, 1, 2, 3], [2, 0, 3, 1]])
@pytest.mark.parametrize("form", ["square", "jittered", "sheared", "inverted", "tiny", "far"])
def test_against_per_point_kernel(E, gpu, nx, ny, order, form):
    mesh = E.Q4block(1.0, 0.7, nx, ny)
    rng = np.random.default_rng(nx)
    xy = mesh.xy.copy()
    if form != "square":
        xy += rng.uniform(-0.2, 0.2, size=xy.shape) * np.array([1.0 / nx, 0.7 / ny])
    if form == "sheared":
        xy = xy @ np.array([[1.0, 0.3], [0.8, 1.0]])
    if form == "inverted":
        xy[:, 0] *= -1.0
    if form == "tiny":
        xy *= 1e-130  # det J is far below 1e-200: reciprocals of extreme exponent
    if form == "far":
        xy += 8.0
    mesh = E.Mesh("Q4", mesh.conn, xy)
    kappa = rng.uniform(0.5, 2.0, mesh.nel)
    (K1, F1), (K0, F0) = both(E, mesh, order, kappa)
    assert np.array_equal(K1.indptr, K0.indptr) and np.array_equal(K1.indices, K0.indices)
    # coordinates far from the origin: the per-point kernel sums whole coordinates (relative size 8 / h)
    scale = 1.0 if form != "far" else 8.0 * max(nx, ny)
    assert np.abs(K1.data - K0.data).max() <= scale * TOL * np.abs(K0.data).max()
    assert np.abs(F1 - F0).max() <= scale * TOL * np.abs(F0).max()
