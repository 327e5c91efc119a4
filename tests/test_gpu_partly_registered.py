"""Host arrays of which only a part is page-locked (cudaHostRegister) (GPU).

A kernel reads a host array in place only where all of it is page-locked (or
where the device reads pageable memory); the registration is that of the last
byte too, not of the first alone.  What the runtime makes of a copy from such an
array is its own business: the call succeeds with the values of ordinary memory,
or reports an error; afterwards the same system assembles as before.
"""
import mmap

import numpy as np
import pytest

from problems import heat_space

pytestmark = pytest.mark.gpu

PAGE = 1 << 16


class Registered:
    """n doubles in fresh pages, [a, b) of which are page-locked."""

    def __init__(self, n, part):
        import torch

        self.rt = torch.cuda.cudart()
        size = (8 * n + PAGE - 1) // PAGE * PAGE
        self.m = mmap.mmap(-1, size + PAGE)
        raw = np.frombuffer(self.m, dtype=np.uint8)
        off = (-raw.ctypes.data) % PAGE
        self.a = raw[off:off + 8 * n].view(np.float64)
        half = size // 2 // PAGE * PAGE
        assert half > 0
        lo, hi = {"first": (0, half), "last": (half, size), "all": (0, size), "none": (0, 0)}[part]
        self.ptr = self.a.ctypes.data + lo if hi > lo else None
        if self.ptr:
            assert int(self.rt.cudaHostRegister(self.ptr, hi - lo, 0)) == 0

    def close(self):
        import torch

        torch.cuda.synchronize()
        if self.ptr:
            assert int(self.rt.cudaHostUnregister(self.ptr)) == 0


@pytest.mark.parametrize("kind", ["T6", "T3", "Q4", "curved"])
@pytest.mark.parametrize("part", ["none", "first", "last", "all"])
def test_conductivities(E, gpu, kind, part):
    block = {"Q4": E.Q4block, "T3": E.T3block}.get(kind, E.T6block)
    fe = {"Q4": E.FEH1_Q4, "T3": E.FEH1_T3}.get(kind, E.FEH1_T6)
    mesh = block(1.0, 1.0, 150, 150)
    if kind == "curved":
        mesh.xy[mesh.conn[0, 4] - 1] += 1e-4
    fesp = heat_space(E, mesh, fe())
    n = E.ndofs(fesp)
    rule = {"kind": "Gauss", "order": 2} if kind == "Q4" else {"npts": 3}
    am = E.start(E.SysmatAssemblerGPU(), n, n)
    kappa = np.random.default_rng(3).uniform(0.5, 2.0, mesh.nel)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, rule), kappa, -6.0)
    want = E.finish(am).data.copy()
    r = Registered(mesh.nel, part)
    r.a[:] = kappa
    try:
        for _ in range(3):
            try:
                am.heat(r.a, -6.0)
                got = E.finish(am).data
            except E.ElfelError:
                assert part in ("first", "last")
                continue
            assert np.array_equal(got, want)
    finally:
        r.close()
    am.heat(kappa, -6.0)
    assert np.array_equal(E.finish(am).data, want)


@pytest.mark.parametrize("part", ["none", "first", "last", "all"])
def test_values_out(E, gpu, part):
    mesh = E.T6block(1.0, 1.0, 310, 310)
    fesp = E.FESpace(float, mesh, E.FEH1_T6())
    E.numberdofs(fesp)
    n = E.ndofs(fesp)
    am = E.start(E.SysmatAssemblerGPU(), n, n)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), 1.0, -6.0)
    want = E.finish(am).data.copy()
    r = Registered(want.size, part)
    N = E._native
    try:
        for _ in range(3):
            am.heat(None, -6.0)
            r.a[:] = -7.0
            try:
                gpu.check(gpu.lib.elfel_sysmat_csc(am._hd.h, None, None, N.ptr(r.a)))
            except E.ElfelError:
                assert part in ("first", "last")
                continue
            assert np.array_equal(r.a, want)
    finally:
        r.close()
    assert np.array_equal(am.csc().data, want)
