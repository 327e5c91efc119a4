"""Re-assembly and download of a large system on a stream of the caller's (elfel_ctx_set_stream) (GPU).

The download follows the work that the caller has queued on that stream, also
where the values of a system of more than 4M nonzeros would leave in two parts,
and an assembly captured into a CUDA graph can be replayed and downloaded.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def big(E, ctx, etype, k):
    mesh = (E.T6block if etype == "T6" else E.T3block)(1.0, 1.0, k, k)
    fesp = E.FESpace(float, mesh, E.FEH1_T6() if etype == "T6" else E.FEH1_T3())
    E.numberdofs(fesp)
    n = E.ndofs(fesp)
    am = E.start(E.SysmatAssemblerGPU(ctx=ctx), n, n)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), 1.0, -6.0)
    nnz = E.finish(am).nnz
    assert nnz >= 1 << 22
    return am, nnz


def download(E, ctx, am, v):
    ctx.check(ctx.lib.elfel_sysmat_csc(am._hd.h, None, None, E._native.ptr(v)))


@pytest.mark.parametrize("etype,k", [("T6", 310), ("T3", 780)])
def test_download_follows_queued_work(E, gpu, etype, k):
    import torch

    ctx = E.Context(0)
    s = torch.cuda.Stream()
    ctx.set_stream(s.cuda_stream)
    am, nnz = big(E, ctx, etype, k)
    v = torch.full((nnz,), -7.0, dtype=torch.float64).pin_memory()
    want = am.csc().data.copy()
    dev = torch.empty(nnz, dtype=torch.float64, device="cuda")
    for step in range(4):
        before = v.clone()
        am.heat(float(step + 2), -6.0)
        with torch.cuda.stream(s):
            torch.cuda._sleep(20_000_000)  # about 10 ms, then the old values are read
            dev.copy_(v, non_blocking=True)
        download(E, ctx, am, v.numpy())
        torch.cuda.synchronize()
        assert torch.equal(dev.cpu(), before), step
        assert np.allclose(v.numpy(), (step + 2) * want, rtol=1e-14, atol=1e-14), step
    ctx.set_stream(None)


@pytest.mark.parametrize("etype,k", [("T6", 310), ("T3", 780), ("T6", 20)])
def test_captured_assembly(E, gpu, etype, k):
    import torch

    ctx = E.Context(0)
    s = torch.cuda.Stream()
    ctx.set_stream(s.cuda_stream)
    if k >= 300:
        am, nnz = big(E, ctx, etype, k)
    else:
        mesh = E.T6block(1.0, 1.0, k, k)
        fesp = E.FESpace(float, mesh, E.FEH1_T6())
        E.numberdofs(fesp)
        am = E.start(E.SysmatAssemblerGPU(ctx=ctx), E.ndofs(fesp), E.ndofs(fesp))
        E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), 1.0, -6.0)
        nnz = E.finish(am).nnz
    for _ in range(3):
        am.heat(None, -6.0)
    v = torch.full((nnz,), -7.0, dtype=torch.float64).pin_memory().numpy()
    download(E, ctx, am, v)
    want, f = v.copy(), am.rhs().copy()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        am.heat(None, -3.0)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    v[:] = -7.0
    download(E, ctx, am, v)
    assert np.array_equal(v, want)
    assert np.allclose(am.rhs(), 0.5 * f, rtol=1e-14, atol=1e-15 * np.abs(f).max())
    ctx.set_stream(None)
