"""SolvePrecond on a device vector when a device allocation fails (dfm2g_debug_fail_alloc, on the host), whichever of
the first call's allocations it is: the call reports it and the vector is still the caller's, bit for bit, although
the sweeps work in it. With memory again the same handle gives the solution of a handle that never went without
(another schedule may run it: 1e-12 relative FP64, 1e-5 FP32)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim,perm", [(3, False), (3, True), (2, False), (1, True)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_vector_survives_a_failed_allocation(gpu, ndim, perm, dtype):
    torch = pytest.importorskip("torch")
    import delfem2_gb300 as D
    a = D.voxel_problem_arrays(7, 6, 5, 0.2, seed=2)
    n, rng = a["np"], np.random.default_rng(ndim)
    ind, psup = a["psup_ind"], a["psup"]
    if perm:  # numbered without order: thin tiles, a warp per chain
        tet = rng.permutation(n).astype(np.uint32)[a["tet"]]
        ind, psup = D.JArray_PSuP_MeshElem(tet, 4, n)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(0.04 * rng.standard_normal(psup.size * ndim * ndim), np.tile(np.eye(ndim).ravel(), n))
    b = torch.from_numpy(rng.standard_normal(n * ndim).astype(dtype)).cuda()

    def handle():
        ilu = D.CPreconditionerILU()
        ilu.SetPattern0(K)
        ilu.CopyValue(K)
        assert ilu.Decompose()
        return ilu

    want = b.clone()
    handle().SolvePrecond(want)
    tol = 1e-12 if dtype is np.float64 else 1e-5
    failures = 0
    for nth in range(1, 64):
        ilu, x = handle(), b.clone()
        assert gpu.dfm2g_debug_fail_alloc(nth) == 0
        try:
            ilu.SolvePrecond(x)
            break  # fewer allocations than nth: the call went through
        except RuntimeError:
            failures += 1
            assert torch.equal(x, b), nth
        finally:
            assert gpu.dfm2g_debug_fail_alloc(0) == 0
        ilu.SolvePrecond(x)
        assert rel_err(x.cpu().numpy(), want.cpu().numpy()) < tol, nth
    assert failures >= 2 and torch.equal(x, want)
