"""elfel_sysmat_csc with some of its arrays left out (GPU): what is asked for is what the full call gives."""
import ctypes

import numpy as np
import pytest

from problems import heat_space

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("which", ["nzval", "colptr", "rowval", "colptr nzval", ""])
def test_partial_csc(E, gpu, pinned, which):
    import torch

    N = E._native
    mesh = E.jitter(E.T6block(1.0, 1.0, 13, 9), 0.01, seed=2)
    fesp = heat_space(E, mesh, E.FEH1_T6())
    n = E.ndofs(fesp)
    am = E.start(E.SysmatAssemblerGPU(), n, n)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), np.linspace(0.5, 2.0, mesh.nel), -6.0)
    K = E.finish(am)
    full = {"colptr": K.indptr + 1, "rowval": K.indices + 1, "nzval": K.data}
    out = {}
    for k in which.split():
        t = torch.full((full[k].size,), -7, dtype=torch.float64 if k == "nzval" else torch.int64)
        out[k] = (t.pin_memory() if pinned else t).numpy()
    p = {k: N.ptr(out[k], N._dp if k == "nzval" else N._i64p) if k in out else None for k in full}
    gpu.check(gpu.lib.elfel_sysmat_csc(am._hd.h, p["colptr"], p["rowval"], p["nzval"]))
    for k in out:
        assert np.array_equal(out[k], full[k]), k
    nnz = ctypes.c_int64()
    gpu.check(gpu.lib.elfel_sysmat_dims(am._hd.h, None, None, ctypes.byref(nnz)))
    assert nnz.value == K.nnz


@pytest.mark.parametrize("kind", ["T6", "T3", "elasticity"])
def test_head_of_the_values(E, gpu, kind):
    """A system of more than 4M nonzeros, whose values are reduced and copied
    in two parts on two streams: every assembly's values arrive whole (the
    staged copy into pageable arrays is the yardstick), also when the
    coefficient changes between assemblies that nothing waits for."""
    import torch

    from problems import elasticity_setup

    N = E._native
    if kind == "elasticity":
        mesh, fesp, bforce, right = elasticity_setup(E, 300, 150)
        n = E.ndofs(fesp)
        am = E.start(E.SysmatAssemblerGPU(), n, n)
        elit, qpit = E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3})
        E.assemble_elasticity(am, elit, qpit, 1.0, 0.3, True, bforce)
        again = lambda s: am.elasticity(s, 0.3, True, bforce)  # noqa: E731
    else:
        k = 310 if kind == "T6" else 780
        mesh = (E.T6block if kind == "T6" else E.T3block)(1.0, 1.0, k, k)
        fesp = E.FESpace(float, mesh, E.FEH1_T6() if kind == "T6" else E.FEH1_T3())
        E.numberdofs(fesp)
        n = E.ndofs(fesp)
        am = E.start(E.SysmatAssemblerGPU(), n, n)
        E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), 1.0, -6.0)
        again = lambda s: am.heat(s, -6.0)  # noqa: E731
    nnz = ctypes.c_int64()
    gpu.check(gpu.lib.elfel_sysmat_dims(am._hd.h, None, None, ctypes.byref(nnz)))
    assert nnz.value >= 1 << 22
    v = torch.full((nnz.value,), -7.0, dtype=torch.float64).pin_memory().numpy()
    for s in (1.0, 3.0, 0.7):
        again(2.0 * s)
        again(s)
        gpu.check(gpu.lib.elfel_sysmat_csc(am._hd.h, None, None, N.ptr(v)))
        assert np.array_equal(v, am.csc().data), s
