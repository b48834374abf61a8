"""Decompose again and again: the rows of a level are factored by warps that only meet through the rows' flags, so the
factors of 25 decompositions of the same values have the same bits, on patterns with many short levels (a voxel block,
its ILU(1)) and with one row a level (a band)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,kind,fill", [(1, "block", 0), (2, "block", 0), (3, "block", 0), (3, "block", 1),
                                            (3, "band", 0)])
def test_same_factors_every_time(gpu, ndim, kind, fill):
    import delfem2_gb300 as D
    if kind == "block":
        a = D.voxel_problem_arrays(17, 16, 15, 0.1, seed=1)
        n, ind, psup = a["np"], a["psup_ind"], a["psup"]
    else:
        n = 600
        nbr = [[j for j in range(max(0, i - 20), min(n, i + 21)) if j != i] for i in range(n)]
        ind = np.concatenate([[0], np.cumsum([len(b) for b in nbr])]).astype(np.uint32)
        psup = np.array([j for b in nbr for j in b], np.uint32)
    rng = np.random.default_rng(ndim)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(0.02 * rng.standard_normal(np.asarray(psup).size * ndim * ndim),
                 np.tile(np.eye(ndim).ravel(), n) + 0.02 * rng.standard_normal(n * ndim * ndim))
    ilu = D.CPreconditionerILU()
    ilu.Initialize_ILUk(K, fill)
    first = None
    for _ in range(25):
        ilu.CopyValue(K)
        assert ilu.Decompose()
        now = ilu.values()
        first = first or now
        assert all(np.array_equal(x, y) for x, y in zip(first, now))
