"""Rounding error of a product's long row (a hub coupled to 2,000 others): eight lanes and a tree add its blocks, not
one lane's chain (csrc/spmv_tma.cuh, kLongest). Root mean square over 64 vectors, in units of |K||x| of the row, for
random terms: about 1.06e-8 FP32 and 2.0e-17 FP64 over eight sums of 250 1x1 blocks (1.85e-8 and 3.6e-17 over two sums
of 1,000), and 2x2 rows below that, as a block's two products are added first; 64 vectors give it within 20%."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = {1: (1.35e-8, 2.6e-17), 2: (1.35e-8, 1.7e-17)}


@pytest.mark.parametrize("ndim", [1, 2])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_error_of_a_long_row(gpu, ndim, dtype):
    import delfem2_gb300 as D
    n = 2001
    rng = np.random.default_rng(ndim)
    ind = np.concatenate([[0], n - 1 + np.arange(n)]).astype(np.uint32)
    psup = np.concatenate([np.arange(1, n), np.zeros(n - 1)]).astype(np.uint32)
    val = rng.standard_normal((psup.size, ndim, ndim))
    dia = np.tile(3.0 * np.eye(ndim), (n, 1, 1))
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(val.ravel(), dia.ravel())
    v, d = val.astype(dtype).astype(np.longdouble)[:n - 1], dia[0].astype(np.longdouble)
    err = []
    for _ in range(64):
        x = rng.standard_normal((n, ndim)).astype(dtype)
        y = np.zeros(n * ndim, dtype)
        K.MatVec(y, 1.0, x.ravel().copy(), 0.0)
        want = np.einsum("kab,kb->a", v, x[1:]) + d @ x[0]
        size = np.einsum("kab,kb->a", abs(v), abs(x[1:])) + abs(d) @ abs(x[0])
        err.append(((y[:ndim] - want) / size).astype(float))
    assert np.sqrt(np.mean(np.square(err))) < BOUND[ndim][0 if dtype is np.float32 else 1]
