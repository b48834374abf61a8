"""Decompose without device memory for the one-launch factorisation's table (its first allocation) or flags (its
second): the level kernels, which need neither, factor instead, nothing half-made is kept, and the next Decompose takes
the one launch again. A failed allocation is a host-side one (dfm2g_debug_fail_alloc). Factors within 1e-12 relative
(3x3: the two paths fuse their sums differently), equal bits for 1x1 and 2x2."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("nth", [1, 2])
def test_decompose_without_memory(gpu, ndim, nth):
    import ctypes as C

    import delfem2_gb300 as D
    from delfem2_gb300 import _native as N
    n, rng = 400, np.random.default_rng(ndim)
    nbr = [[j for j in range(max(0, i - 4), min(n, i + 5)) if j != i] for i in range(n)]
    ind = np.concatenate([[0], np.cumsum([len(a) for a in nbr])]).astype(np.uint32)
    psup = np.array([j for a in nbr for j in a], np.uint32)
    vc = 0.1 * rng.standard_normal(psup.size * ndim * ndim)
    vd = np.tile(np.eye(ndim).ravel(), n) * 4.0 + 0.1 * rng.standard_normal(n * ndim * ndim)

    def launches():
        c = C.c_ulonglong(0)
        assert gpu.dfm2g_launch_count(C.byref(c)) == N.OK
        return c.value

    def factors(fail):
        ilu.CopyValue(K)
        assert gpu.dfm2g_debug_fail_alloc(fail) == N.OK
        c = launches()
        try:
            assert ilu.Decompose()
        finally:
            assert gpu.dfm2g_debug_fail_alloc(0) == N.OK
        return ilu.values(), launches() - c

    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(vc, vd)
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    by_levels, many = factors(nth)
    at_once, two = factors(0)  # builds the table: one launch more than the next
    again, one = factors(0)
    assert one == 1 and two == 2 and many != one
    for got in (at_once, again):
        for a, b in zip(got, by_levels):
            assert np.array_equal(a, b) if ndim < 3 else rel_err(a, b) < 1e-12
