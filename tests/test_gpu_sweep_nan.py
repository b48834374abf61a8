"""A NaN in a sweep's right-hand side gives NaN rows whatever its payload, in every schedule that marks rows not yet
written by an all-ones NaN: FP64 arithmetic hands a payload on, so the marker itself (and its negation 0x7fff...f) as
an input must not come out of a row as the marker, which its dependents would wait for until their time is up. The same
rows are NaN as for the plain quiet NaN (and as in the level schedule, which marks nothing), all others have the same
bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PAYLOADS = [0xFFFFFFFFFFFFFFFF, 0x7FFFFFFFFFFFFFFF, 0x7FF8000000000001]


def _handle(ndim):
    import delfem2_gb300 as D
    a = D.voxel_problem_arrays(5, 4, 6, 0.2, seed=2)
    n, rng = a["np"], np.random.default_rng(ndim)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(a["psup_ind"], a["psup"])
    K.set_values(0.04 * rng.standard_normal(a["psup"].size * ndim * ndim), np.tile(np.eye(ndim).ravel(), n))
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    return ilu, n, rng


@pytest.mark.parametrize("ndim,mode", [(1, 0), (1, 5), (2, 0), (2, 7)] + [(3, m) for m in (0, 3, 4, 5, 6, 8)])
def test_nan_of_any_payload(gpu, ndim, mode):
    ilu, n, rng = _handle(ndim)
    b = rng.standard_normal(n * ndim)
    at = ndim * (n // 2) + ndim - 1  # rows of either sweep before and after it
    for sweep in (ilu.ForwardSubstitution, ilu.BackwardSubstitution, ilu.SolvePrecond):
        by_levels, want = b.copy(), b.copy()
        by_levels[at] = want[at] = np.nan
        ilu.set_sweep_mode(1)  # a launch per level: no markers
        sweep(by_levels)
        ilu.set_sweep_mode(mode)
        sweep(want)
        assert np.isnan(want).any() and np.array_equal(np.isnan(want), np.isnan(by_levels))
        for payload in PAYLOADS:
            x = b.copy()
            x.view(np.uint64)[at] = payload
            sweep(x)
            assert np.array_equal(np.isnan(x), np.isnan(want))
            ok = ~np.isnan(want)
            assert np.array_equal(x[ok], want[ok])
