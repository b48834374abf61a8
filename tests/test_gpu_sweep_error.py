"""Rounding error of the FP64 sweeps (csrc/tile_kernel.cuh) against the same recurrences in long double, as a relative
norm over a 13 x 12 x 11 voxel block's rows. A row whose finished sum is subtracted from its right-hand side rounds
once at the result's size (0.45 of 2^-53 root mean square, 0.5e-16) and otherwise at its sum's: 0.5e-16 to 0.9e-16 over
these systems for 1x1 to 3x3 blocks. A chain of products started from the right-hand side rounds at its size in every
product, 1.0e-16 to 1.8e-16, and is outside the bounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = {1: 0.8e-16, 2: 1.2e-16, 3: 1.2e-16}


def _factored(ndim, seed):
    import delfem2_gb300 as D
    a = D.voxel_problem_arrays(13, 12, 11, 1.0 / 13, seed=seed, e_range=(0.1, 10.0))
    if ndim == 3:  # the elastic block itself
        P = D.StaticElasticProblem(a)
        P.assemble()
        assert P.factor()
        return P.ilu, P
    n, bb = a["np"], ndim * ndim
    rng = np.random.default_rng(seed)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(a["psup_ind"], a["psup"])
    K.set_values(0.05 * rng.standard_normal(a["psup"].size * bb),
                 np.tile(np.eye(ndim).ravel(), n) + 0.05 * rng.standard_normal(n * bb))
    ilu = D.CPreconditionerILU()
    ilu.SetPattern0(K)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    return ilu, K


def _forward(rs, col, dia, vc, vd, b):
    z = np.zeros_like(b)
    for i in range(b.shape[0]):
        s = slice(rs[i], dia[i])
        z[i] = vd[i] @ (b[i] - np.einsum("kab,kb->a", vc[s], z[col[s]]))
    return z


def _backward(rs, col, dia, vc, b):
    z = np.zeros_like(b)
    for i in range(b.shape[0] - 1, -1, -1):
        s = slice(dia[i], rs[i + 1])
        z[i] = b[i] - np.einsum("kab,kb->a", vc[s], z[col[s]])
    return z


@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_error_of_the_fp64_sweeps(gpu, ndim):
    err = []
    for seed in range(3):
        ilu, keep = _factored(ndim, seed)
        rs = np.asarray(ilu.row_start()).astype(np.int64)
        col, dia = (np.asarray(a).astype(np.int64) for a in ilu.pattern())
        vc, vd = (np.asarray(a).astype(np.longdouble).reshape(-1, ndim, ndim) for a in ilu.values())
        b = np.random.default_rng(seed).standard_normal((rs.size - 1, ndim))
        want_f, want_b = _forward(rs, col, dia, vc, vd, b.astype(np.longdouble)), _backward(
            rs, col, dia, vc, b.astype(np.longdouble))
        f, g = b.ravel().copy(), b.ravel().copy()
        ilu.ForwardSubstitution(f)
        ilu.BackwardSubstitution(g)
        err.append([float(np.linalg.norm((x - w.ravel()).astype(float)) / np.linalg.norm(w.astype(float)))
                    for x, w in ((f, want_f), (g, want_b))])
    assert (np.mean(err, 0) < BOUND[ndim]).all(), err
