"""Pattern build, column by column (GPU): one thread per column (sort_cols_k) against the warp's column sorts and scipy.

Columns of every length around the register networks' sizes (6, 12, 18, 24, 36,
40), the batch of 32 columns, up to 16 and 32 column groups and more, and row
spans around 26 and 25 bits.  Integers are equal; values sum in the order of the triplets,
so they are equal bit for bit to a sequential sum.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 5, 6, 7, 12, 13, 18, 19, 24, 25, 36, 37, 40, 41, 64, 65, 256, 300]


def expected(I, J, V, nrow, ncol):
    """CSC of triplets with duplicates summed left to right."""
    order = np.lexsort((np.arange(I.size), I, J))
    i, j, v = I[order], J[order], V[order]
    new = np.r_[True, (i[1:] != i[:-1]) | (j[1:] != j[:-1])] if i.size else np.zeros(0, bool)
    pos = np.cumsum(new) - 1
    x = np.zeros(int(new.sum()))
    x[pos[new]] = v[new]
    rest = np.flatnonzero(~new)
    np.add.at(x, pos[rest], v[rest])  # unbuffered, in order
    colptr = np.zeros(ncol + 1, dtype=np.int64)
    np.add.at(colptr, j[new], 1)  # j is 1-based: counts of column j at j
    return np.cumsum(colptr), i[new], x


@pytest.mark.parametrize("rows", ["few", "wide"])
@pytest.mark.parametrize("ncol", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("n", LENGTHS)
def test_triplets(E, gpu, n, ncol, rows):
    rng = np.random.default_rng(n * 1000 + ncol)
    nrow = max(1, n // 2) if rows == "few" else 2_000_000_000
    lens = np.full(ncol, n)
    lens[::7] = rng.integers(0, n + 1, lens[::7].size)
    J = np.repeat(np.arange(1, ncol + 1), lens)
    I = rng.integers(1, nrow + 1, J.size)
    if rows == "wide" and I.size:
        I[rng.integers(0, I.size, I.size // 2)] = 1  # duplicates
    p = rng.permutation(J.size)
    I, J = I[p], J[p]
    V = rng.standard_normal(I.size)
    ctx = E.default_context()
    N = E._native if hasattr(E, "_native") else __import__("importlib").import_module(E.__name__ + "._native")
    h = ctypes.c_void_p()
    ctx.check(ctx.lib.elfel_sysmat_create(ctx.h, ctypes.byref(h)))
    try:
        ctx.check(ctx.lib.elfel_sysmat_start(h, nrow, ncol))
        ctx.check(ctx.lib.elfel_sysmat_assemble_coo(h, N.ptr(I, N._i64p), N.ptr(J, N._i64p), N.ptr(V), I.size))
        nnz = ctypes.c_int64()
        ctx.check(ctx.lib.elfel_sysmat_finish(h, ctypes.byref(nnz)))
        cp, rv, x = np.zeros(ncol + 1, np.int64), np.zeros(max(nnz.value, 1), np.int64), np.zeros(max(nnz.value, 1))
        ctx.check(ctx.lib.elfel_sysmat_csc(h, N.ptr(cp, N._i64p), N.ptr(rv, N._i64p), N.ptr(x)))
    finally:
        ctx.lib.elfel_sysmat_destroy(h)
    ecp, erv, ex = expected(I, J, V, nrow, ncol)
    assert np.array_equal(cp - 1, ecp)
    assert nnz.value == erv.size
    assert np.array_equal(rv[: nnz.value], erv)
    assert np.array_equal(x[: nnz.value], ex)


@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, (1 << 18) + 333])
@pytest.mark.parametrize("pinned", [False, True])
def test_values_behind_the_indices(E, gpu, n, pinned):
    """From 2^18 triplets on the pattern is built while the values are uploaded: one
    and two appends, finish! twice, an index out of range, and a new start!."""
    import torch

    rng = np.random.default_rng(n)
    ndof = 20000
    host = lambda a: torch.from_numpy(a).pin_memory().numpy() if pinned else a  # noqa: E731
    I, J = (host(rng.integers(1, ndof + 1, n)) for _ in range(2))
    V = host(rng.standard_normal(n))
    ctx = E.default_context()
    N = __import__("importlib").import_module(E.__name__ + "._native")
    L, ip = ctx.lib, lambda a: N.ptr(a, N._i64p)  # noqa: E731
    h = ctypes.c_void_p()
    ctx.check(L.elfel_sysmat_create(ctx.h, ctypes.byref(h)))

    def append(sl):
        i, j, v = I[sl], J[sl], V[sl]
        ctx.check(L.elfel_sysmat_assemble_coo(h, ip(i), ip(j), N.ptr(v), i.size))

    def result():
        nnz = ctypes.c_int64()
        ctx.check(L.elfel_sysmat_finish(h, ctypes.byref(nnz)))
        cp, rv, x = np.zeros(ndof + 1, np.int64), np.zeros(nnz.value, np.int64), np.zeros(nnz.value)
        ctx.check(L.elfel_sysmat_csc(h, ip(cp), ip(rv), N.ptr(x)))
        return cp - 1, rv, x

    try:
        want = expected(I, J, V, ndof, ndof)
        for cuts in ([0, n], [0, 1000, n], [0, n - 10, n]):
            ctx.check(L.elfel_sysmat_start(h, ndof, ndof))
            for a, b in zip(cuts[:-1], cuts[1:]):
                append(slice(a, b))
            for _ in range(2):
                assert all(np.array_equal(p, q) for p, q in zip(result(), want))
            append(slice(0, 500))  # append after finish!
            again = expected(*(np.r_[a, a[:500]] for a in (I, J, V)), ndof, ndof)
            assert all(np.array_equal(p, q) for p, q in zip(result(), again))
        wrong = host(np.full(7, ndof + 1))
        ctx.check(L.elfel_sysmat_assemble_coo(h, ip(wrong), ip(J[:7]), N.ptr(V[:7]), 7))
        nnz = ctypes.c_int64()
        assert L.elfel_sysmat_finish(h, ctypes.byref(nnz)) != 0
        ctx.check(L.elfel_sysmat_start(h, ndof, ndof))
        append(slice(0, n))
        assert all(np.array_equal(p, q) for p, q in zip(result(), want))
    finally:
        L.elfel_sysmat_destroy(h)


def fused(E, dofs, ndofs, conn, xy):
    """K of the heat form on T3 elements with the given element DOFs."""
    N = __import__("importlib").import_module(E.__name__ + "._native")
    ctx = E.default_context()
    h = ctypes.c_void_p()
    ctx.check(ctx.lib.elfel_sysmat_create(ctx.h, ctypes.byref(h)))
    try:
        ip = lambda a: N.ptr(a, N._i64p)  # noqa: E731
        u = N.Space(3, 1, conn.shape[0], xy.shape[0], ip(conn), N.ptr(xy), ip(dofs))
        pc, w = np.array([[1 / 3, 1 / 3]]), np.array([0.5])
        d = N.FusedDesc(N.ELFEL_HEAT, 1, N.ptr(pc), N.ptr(w), ndofs, u, N.Space(), N.ELFEL_SHAPE_TRIANGLE, 2)
        ctx.check(ctx.lib.elfel_fused_setup(h, ctypes.byref(d)))
        kappa = np.ones(conn.shape[0])
        ctx.check(ctx.lib.elfel_fused_heat(h, N.ptr(kappa), 0.0))
        nnz = ctypes.c_int64()
        ctx.check(ctx.lib.elfel_sysmat_dims(h, None, None, ctypes.byref(nnz)))
        cp, rv, x = np.zeros(ndofs + 1, np.int64), np.zeros(nnz.value, np.int64), np.zeros(nnz.value)
        ctx.check(ctx.lib.elfel_sysmat_csc(h, ip(cp), ip(rv), N.ptr(x)))
        F = np.zeros(ndofs)
        ctx.check(ctx.lib.elfel_sysmat_rhs(h, N.ptr(F)))
    finally:
        ctx.lib.elfel_sysmat_destroy(h)
    return cp - 1, rv, x


def t3_triplets(dofs):
    n = dofs.shape[0]
    I = np.repeat(dofs[:, None, :], 3, axis=1).ravel()
    J = np.repeat(dofs[:, :, None], 3, axis=2).ravel()
    k = np.array([[1.0, -0.5, -0.5], [-0.5, 0.5, 0.0], [-0.5, 0.0, 0.5]])
    return I, J, np.tile(k.ravel(), n)


@pytest.mark.parametrize("share", [1, 2, 3, 8, 9, 15, 16, 17, 24, 31, 32, 40, 120])
@pytest.mark.parametrize("repeat", [False, True])
def test_shared_dofs(E, gpu, share, repeat):
    """Unit right triangles whose DOFs are shared by `share` elements each, with and
    without elements that hold one DOF twice."""
    rng = np.random.default_rng(share)
    nel = 400
    ndofs = max(3, 3 * nel // share)
    dofs = np.stack([rng.permutation(ndofs)[:3] for _ in range(nel)]) + 1
    if repeat:
        dofs[::5, 2] = dofs[::5, 0]
    dofs = np.ascontiguousarray(dofs, dtype=np.int64)
    xy = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
    conn = np.tile(np.array([[1, 2, 3]], dtype=np.int64), (nel, 1))
    cp, rv, x = fused(E, dofs, ndofs, conn, xy)
    ecp, erv, ex = expected(*t3_triplets(dofs), ndofs, ndofs)
    assert np.array_equal(cp, ecp) and np.array_equal(rv, erv)
    assert np.array_equal(x, ex)  # multiples of 1/2: sums are exact


@pytest.mark.parametrize("span", [(1 << 26) - 2, (1 << 26) - 1, (1 << 26) + 5])
def test_row_span(E, gpu, span):
    """DOF numbers on both sides of the span that fits a 32-bit key."""
    ndofs = span + 1
    dofs = np.array([[1, 2, ndofs], [2, 40, ndofs], [1, ndofs, 40], [3, 4, 5]], dtype=np.int64)
    xy = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
    conn = np.tile(np.array([[1, 2, 3]], dtype=np.int64), (4, 1))
    cp, rv, x = fused(E, dofs, ndofs, conn, xy)
    ecp, erv, ex = expected(*t3_triplets(dofs), ndofs, ndofs)
    assert np.array_equal(cp, ecp) and np.array_equal(rv, erv) and np.array_equal(x, ex)
