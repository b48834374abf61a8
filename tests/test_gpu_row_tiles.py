"""Row products in tiles (csrc/spmv_tma.cuh) and the reductions of the solvers around them, where their layout turns
over: 40, 80 and 150 rows (a tile's least and most), 1,365 and 1,366 rows of 3x3 blocks (4,096 elements: one CTA's
reduction), 6,080 and 12,160 rows (one tile for each of 152 SMs), rows without a block, and one row at and above the
most blocks a tile holds. Against the same product in long double: a row of k blocks sums at most 3 k + 3 products, so
its error is below (3 k + 8) eps |K| |x|. The solves are of diagonally dominant systems to 1e-10 (true residual)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, ndim, long_row=0, seed=0):
    """A symmetric pattern of random short links (plus one row with `long_row` blocks), symmetric dominant values."""
    rng = np.random.default_rng(1000 * n + ndim + seed)
    if n > 1:
        k = min(4, n - 1)
        a = rng.integers(0, n, k * n)
        b = (a + rng.integers(1, min(n, 60), a.size)) % n
        if long_row:
            a, b = np.concatenate([a, np.zeros(long_row, int)]), np.concatenate([b, 1 + np.arange(long_row)])
            keep = ((a != 0) & (b != 0)) | (np.arange(a.size) >= k * n)
            a, b = a[keep], b[keep]
        i, j = np.minimum(a, b), np.maximum(a, b)
        i, j = np.unique(np.stack([i[i != j], j[i != j]]), axis=1)
    else:
        i = j = np.zeros(0, int)
    w = rng.standard_normal((i.size, ndim, ndim))
    row, col = np.concatenate([i, j]), np.concatenate([j, i])
    val = np.concatenate([w, w.transpose(0, 2, 1)])
    o = np.lexsort((col, row))
    row, col, val = row[o], col[o], val[o]
    ind = np.searchsorted(row, np.arange(n + 1)).astype(np.uint32)
    dom = np.zeros(n)
    np.add.at(dom, row, np.abs(val).sum((1, 2)))
    dia = np.eye(ndim)[None] * (dom + 1.0)[:, None, None]
    return ind, col.astype(np.uint32), row, val, dia


def _matrix(ind, col, val, dia, ndim):
    import delfem2_gb300 as D
    K = D.CMatrixSparse()
    K.Initialize(ind.size - 1, ndim, True)
    K.SetPattern(ind, col)
    K.set_values(val.ravel(), dia.ravel())
    return K


def _check_product(K, ind, col, row, val, dia, ndim):
    n = ind.size - 1
    for dt, eps in ((np.float64, 2.0 ** -53), (np.float32, 2.0 ** -24)):
        x = np.random.default_rng(5).standard_normal((n, ndim)).astype(dt)
        v, d = val.astype(dt).astype(np.longdouble), dia.astype(dt).astype(np.longdouble)
        ex, nr = np.einsum("iab,ib->ia", d, x), np.einsum("iab,ib->ia", abs(d), abs(x))
        np.add.at(ex, row, np.einsum("kab,kb->ka", v, x[col]))
        np.add.at(nr, row, np.einsum("kab,kb->ka", abs(v), abs(x[col])))
        y = np.zeros(n * ndim, dt)
        K.MatVec(y, 1.0, x.ravel().copy(), 0.0)
        bound = (ndim * np.diff(ind.astype(np.int64)) + 8)[:, None] * eps * nr
        assert (np.abs(y.reshape(n, ndim) - ex) <= bound).all()


@pytest.mark.parametrize("n", [1, 2, 39, 40, 41, 80, 81, 150, 151, 1365, 1366, 6080, 6081, 12161, 24001])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_row_products(gpu, n, ndim):
    s = _system(n, ndim)
    _check_product(_matrix(s[0], s[1], s[3], s[4], ndim), *s, ndim)


@pytest.mark.parametrize("blocks", [1152, 1153, 1424, 1425, 2304, 2305])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_row_products_long_row(gpu, blocks, ndim):
    s = _system(2400, ndim, blocks)
    _check_product(_matrix(s[0], s[1], s[3], s[4], ndim), *s, ndim)


@pytest.mark.parametrize("n", [1, 40, 41, 1365, 1366, 4097, 6081])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_solves(gpu, n, ndim):
    import delfem2_gb300 as D
    s = _system(n, ndim)
    ind, col, row, val, dia = s
    K = _matrix(ind, col, val, dia, ndim)
    ilu = D.CPreconditionerILU()
    ilu.Initialize_ILUk(K, 0)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    b = np.random.default_rng(9).standard_normal(n * ndim)

    def rel(x):
        X = x.reshape(n, ndim)
        y = np.einsum("iab,ib->ia", dia, X)
        np.add.at(y, row, np.einsum("kab,kb->ka", val, X[col]))
        return np.linalg.norm(y.ravel() - b) / np.linalg.norm(b)

    x = np.zeros(n * ndim)
    D.Solve_PCG(b.copy(), x, 1e-11, 200, K, ilu)
    assert rel(x) < 1e-10
    x = np.zeros(n * ndim)
    D.Solve_CG(b.copy(), x, 1e-11, 400, K)
    assert rel(x) < 1e-10
    x = np.zeros(n * ndim)
    D.Solve_PCG_Mixed(b.copy(), x, 1e-11, K, ilu, method="reliable")
    assert rel(x) < 1e-10


@pytest.mark.parametrize("n", [1, 41, 1366])
@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_precond_of_a_device_vector(gpu, n, ndim, offset):
    """SolvePrecond works straight in a device vector that starts on 16 bytes and through a copy in one that does not:
    the same bits as the host vector's call either way, and nothing written beside the vector."""
    torch = pytest.importorskip("torch")
    import delfem2_gb300 as D
    ind, col, row, val, dia = _system(n, ndim)
    ilu = D.CPreconditionerILU()
    K = _matrix(ind, col, val, dia, ndim)
    ilu.Initialize_ILUk(K, 0)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    for dt in (np.float64, np.float32):
        b = np.random.default_rng(4).standard_normal(n * ndim).astype(dt)
        want = b.copy()
        ilu.SolvePrecond(want)
        room = torch.full((n * ndim + 8,), 7.0, dtype=getattr(torch, dt.__name__), device="cuda")
        vec = room[offset:offset + n * ndim]
        vec.copy_(torch.from_numpy(b))
        ilu.SolvePrecond(vec)
        assert np.array_equal(vec.cpu().numpy(), want)
        assert (room[:offset] == 7.0).all() and (room[offset + n * ndim:] == 7.0).all()
