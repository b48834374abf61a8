"""The kernels that ordinary patterns do not reach: the factorisation by levels (rows too long for the one-launch kernel's
shared memory), a warp per chain in the sweeps (rows of more than 15 blocks in a triangle), and the row products with
eight lanes or a warp a row (a row of more than 16 blocks, 1,152 for 3x3) inside every solver. Each test shows by the
launch count or dfm2g_ilu_last_kernel, or by the rule's own limit on both sides, that it is there. Factors within
1e-10 of the oracle's (3x3; equal bits for 1x1 and 2x2), sweeps within 1e-12 FP64 and 1e-5 FP32, products within
(ndim k + 8) eps |K||x| of a k-block row, solves of diagonally dominant systems to 1e-10."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
CHAINS = 5


def _banded(n, width):
    nbr = [[j for j in range(max(0, i - width), min(n, i + width + 1)) if j != i] for i in range(n)]
    return np.concatenate([[0], np.cumsum([len(a) for a in nbr])]).astype(np.uint32), np.array(
        [j for a in nbr for j in a], np.uint32)


def _runs(n, seed):
    """Runs of (i - 1, i) couplings, cut at random, and nine couplings a row to anywhere."""
    rng = np.random.default_rng(seed)
    i = np.arange(1, n)[rng.random(n - 1) < 0.9]
    a = np.concatenate([i, np.repeat(np.arange(n), 9)])
    b = np.concatenate([i - 1, rng.integers(0, n, 9 * n)])
    a, b = a[a != b], b[a != b]
    key = np.unique(np.concatenate([a * n + b, b * n + a]))
    return np.searchsorted(key // n, np.arange(n + 1)).astype(np.uint32), (key % n).astype(np.uint32)


def _handles(ind, psup, ndim, seed, off=0.3):
    import delfem2_gb300 as D
    n, rng = ind.size - 1, np.random.default_rng(seed)
    vc = off * rng.standard_normal(psup.size * ndim * ndim) / np.sqrt(psup.size / n)
    vd = np.tile(np.eye(ndim).ravel(), n) * 4.0 + 0.1 * rng.standard_normal(n * ndim * ndim)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(vc, vd)
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    ilu.CopyValue(K)
    return K, ilu, vc, vd


def _factors(port, ind, psup, ndim, vc, vd):
    rs, col, dia = port.ilu_pattern_k(ind, psup, 0)
    ivc, ivd = port.nd_ilu_copy_value(ndim, ind, psup, vc, vd, 0, rs, col)
    st, ivc, ivd = port.nd_ilu_decompose(ndim, rs, col, dia, ivc, ivd)
    assert st == 0
    return rs, col, dia, ivc, ivd


# a row's shared memory, blocks and table: 72 (2 w + 1) + 2 w^2 bytes for 3x3 (32 for 2x2, 8 for 1x1), at most 51,200
@pytest.mark.parametrize("ndim,width,by_levels", [(1, 150, False), (1, 160, True), (2, 135, False), (2, 150, True),
                                                  (3, 120, False), (3, 130, True)])
def test_factor_of_long_rows(gpu, port, ndim, width, by_levels):
    from delfem2_gb300 import _native as N
    ind, psup = _banded(330, width)
    K, ilu, vc, vd = _handles(ind, psup, ndim, width)
    c = [C.c_ulonglong(0), C.c_ulonglong(0)]
    assert gpu.dfm2g_launch_count(C.byref(c[0])) == N.OK
    assert ilu.Decompose() and ilu.n_singular == 0
    assert gpu.dfm2g_launch_count(C.byref(c[1])) == N.OK
    assert c[1].value - c[0].value == (330 if by_levels else 2)  # a launch per level; or the table and the rows
    _, _, _, ivc, ivd = _factors(port, ind, psup, ndim, vc, vd)
    gvc, gvd = ilu.values()
    if ndim == 3:
        assert rel_err(gvd, ivd) < 1e-10 and rel_err(gvc, ivc) < 1e-10
    else:
        assert np.array_equal(gvc, ivc) and np.array_equal(gvd, ivd)


def _check_sweeps(port, ilu, o, ndim):
    rs, col, dia, ivc, ivd = o
    v = np.random.default_rng(3).standard_normal((rs.size - 1) * ndim)
    fo = port.nd_ilu_forward(ndim, rs, col, dia, ivc, ivd, v)
    go = port.nd_ilu_backward(ndim, rs, col, dia, ivc, fo)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        f, g, z = v.astype(dtype), fo.astype(dtype), v.astype(dtype)
        ilu.ForwardSubstitution(f)
        ilu.BackwardSubstitution(g)
        ilu.SolvePrecond(z)
        assert rel_err(f, fo) < tol and rel_err(g, go) < tol and rel_err(z, go) < tol
        assert [ilu.last_kernel(dtype is np.float64, b) for b in (False, True)] == [CHAINS, CHAINS]


@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("kind", ["band", "runs"])
def test_chains_of_long_rows(gpu, port, ndim, kind):
    """One chain through all rows, every dependency in it; and chains cut at random among dependencies everywhere."""
    ind, psup = _banded(400, 18) if kind == "band" else _runs(1500, ndim)
    K, ilu, vc, vd = _handles(ind, psup, ndim, 7)
    assert ilu.Decompose()
    _check_sweeps(port, ilu, _factors(port, ind, psup, ndim, vc, vd), ndim)


@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_chain_kernel_shared_by_two_record_sizes(gpu, port, ndim):
    """Longer records, shorter ones, the longer again: the shorter must not lower the kernel's shared-memory limit."""
    pair = []
    for width in (30, 17):
        ind, psup = _banded(300, width)
        K, ilu, vc, vd = _handles(ind, psup, ndim, width)
        assert ilu.Decompose()
        pair.append((ilu, _factors(port, ind, psup, ndim, vc, vd), K))
    for ilu, o, _ in (pair[0], pair[1], pair[0]):
        _check_sweeps(port, ilu, o, ndim)


def _hub(n, ndim, blocks, seed=0):
    """A symmetric dominant system of short rows with row 0 coupled to `blocks` others."""
    rng = np.random.default_rng(seed + blocks)
    i, j = np.concatenate([np.arange(1, n - 1), np.zeros(blocks, int)]), np.concatenate(
        [np.arange(2, n), np.linspace(1, n - 1, blocks).astype(int)])
    w = rng.standard_normal((i.size, ndim, ndim)) / np.sqrt(blocks)
    row, col = np.concatenate([i, j]), np.concatenate([j, i])
    val = np.concatenate([w, w.transpose(0, 2, 1)])
    o = np.lexsort((col, row))
    row, col, val = row[o], col[o], val[o]
    dom = np.zeros(n)
    np.add.at(dom, row, np.abs(val).sum((1, 2)))
    dia = np.eye(ndim)[None] * (dom + 1.0)[:, None, None]
    return np.searchsorted(row, np.arange(n + 1)).astype(np.uint32), col.astype(np.uint32), row, val, dia


@pytest.mark.parametrize("ndim,blocks", [(1, 16), (1, 17), (1, 700), (2, 16), (2, 17), (2, 700), (3, 1152), (3, 1153)])
def test_solves_with_a_long_row(gpu, ndim, blocks):
    import delfem2_gb300 as D
    n = 1500
    ind, col, row, val, dia = _hub(n, ndim, blocks)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, col)
    K.set_values(val.ravel(), dia.ravel())
    for dtype, eps in ((np.float64, 2.0 ** -53), (np.float32, 2.0 ** -24)):
        x = np.random.default_rng(5).standard_normal((n, ndim)).astype(dtype)
        v, d = val.astype(dtype).astype(np.longdouble), dia.astype(dtype).astype(np.longdouble)
        want, size = np.einsum("iab,ib->ia", d, x), np.einsum("iab,ib->ia", abs(d), abs(x))
        np.add.at(want, row, np.einsum("kab,kb->ka", v, x[col]))
        np.add.at(size, row, np.einsum("kab,kb->ka", abs(v), abs(x[col])))
        y = np.zeros(n * ndim, dtype)
        K.MatVec(y, 1.0, x.ravel().copy(), 0.0)
        bound = (ndim * np.diff(ind.astype(np.int64)) + 8)[:, None] * eps * size
        assert (np.abs(y.reshape(n, ndim) - want) <= bound).all()
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    b = np.random.default_rng(9).standard_normal(n * ndim)

    def rel(x):
        X = x.reshape(n, ndim)
        y = np.einsum("iab,ib->ia", dia, X)
        np.add.at(y, row, np.einsum("kab,kb->ka", val, X[col]))
        return np.linalg.norm(y.ravel() - b) / np.linalg.norm(b)

    for solve in (lambda x: D.Solve_PCG(b.copy(), x, 1e-11, 300, K, ilu),
                  lambda x: D.Solve_CG(b.copy(), x, 1e-11, 1000, K),
                  lambda x: D.Solve_PBiCGStab(b.copy(), x, 1e-11, 300, K, ilu),
                  lambda x: D.Solve_PCG_Mixed(b, x, 1e-11, K, ilu, method="reliable"),
                  lambda x: D.Solve_PCG_Mixed(b, x, 1e-11, K, ilu, method="restart")):
        x = np.zeros(n * ndim)
        solve(x)
        assert rel(x) < 1e-10
