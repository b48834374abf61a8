"""The one-launch factorisation (k_ilu_factor_flow, csrc/ilu.cu) where its layout turns over, against the oracle:
rows without dependencies, row triangles of 1, 7, 31-33 and 70 blocks (the readiness mask takes 32 rows at a time;
the register rounds end at 7 and 14 blocks of 3x3), one row per level, a row too long for shared memory (one launch
per level), repeated decompositions of one handle with other values, and singular pivots. Tolerance 1e-10 relative
for 3x3 factors (sums fused differently than the oracle's), bit equality for 1x1 and 2x2."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _banded(n, width):
    nbr = [[j for j in range(max(0, i - width), min(n, i + width + 1)) if j != i] for i in range(n)]
    ind = np.concatenate([[0], np.cumsum([len(a) for a in nbr])]).astype(np.uint32)
    return ind, np.array([j for a in nbr for j in a] or [0], np.uint32)[: ind[-1]]


def _handles(ind, psup, ndim):
    import delfem2_gb300 as D
    K = D.CMatrixSparse()
    K.Initialize(ind.size - 1, ndim, True)
    K.SetPattern(ind, psup)
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    return K, ilu


def _values(rng, n, nnz, ndim):
    vc = 0.3 * rng.standard_normal(nnz * ndim * ndim) / max(1.0, np.sqrt(nnz / n))
    return vc, np.tile(np.eye(ndim).ravel(), n) * 4.0 + 0.1 * rng.standard_normal(n * ndim * ndim)


@pytest.mark.parametrize("n,width", [(1, 0), (40, 0), (300, 1), (150, 7), (80, 31), (80, 32), (80, 33), (200, 70)])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_factor_rows(gpu, port, n, width, ndim):
    ind, psup = _banded(n, width)
    K, ilu = _handles(ind, psup, ndim)
    for seed in (1, 2):  # the second decomposition of one handle
        vc, vd = _values(np.random.default_rng(seed), n, psup.size, ndim)
        K.set_values(vc, vd)
        ilu.CopyValue(K)
        assert ilu.Decompose() and ilu.n_singular == 0
        rs, col, dia = port.ilu_pattern_k(ind, psup, 0)
        ivc, ivd = port.nd_ilu_copy_value(ndim, ind, psup, vc, vd, 0, rs, col)
        st, ivc, ivd = port.nd_ilu_decompose(ndim, rs, col, dia, ivc, ivd)
        assert st == 0
        gvc, gvd = ilu.values()
        if ndim == 3:
            assert rel_err(gvd, ivd) < 1e-10 and (psup.size == 0 or rel_err(gvc, ivc) < 1e-10)
        else:
            assert np.array_equal(gvc, ivc) and np.array_equal(gvd, ivd)


@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_singular_pivots_are_counted(gpu, ndim):
    n = 20
    ind, psup = _banded(n, 0)
    K, ilu = _handles(ind, psup, ndim)
    vd = np.tile(np.eye(ndim).ravel(), n)
    vd.reshape(n, -1)[:3] = 0.0
    K.set_values(np.zeros(0), vd)
    ilu.CopyValue(K)
    assert ilu.Decompose() and ilu.n_singular == 3
    assert np.array_equal(ilu.values()[1], vd)  # identity inverted, zero pivots left
