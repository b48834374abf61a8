"""A 1x1 or 2x2 MatVec of device vectors is queued and returns: it can be captured into a CUDA graph (nothing in it
waits for the device) and a replay multiplies what the vectors hold by then. Same bits as the call outside a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", [1, 2])
@pytest.mark.parametrize("n", [1, 700, 20_001])
def test_matvec_is_captured(gpu, ndim, n):
    torch = pytest.importorskip("torch")
    import delfem2_gb300 as D
    rng = np.random.default_rng(n)
    nbr = [[j for j in (i - 2, i - 1, i + 1) if 0 <= j < n] for i in range(n)]
    ind = np.concatenate([[0], np.cumsum([len(a) for a in nbr])]).astype(np.uint32)
    psup = np.array([j for a in nbr for j in a], np.uint32)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(rng.standard_normal(psup.size * ndim * ndim), rng.standard_normal(n * ndim * ndim))
    for dtype in (torch.float64, torch.float32):
        x = torch.randn(n * ndim, dtype=dtype, device="cuda")
        want, y = torch.zeros_like(x), torch.zeros_like(x)
        K.MatVec(y, 1.0, x, 0.0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            K.MatVec(y, 1.0, x, 0.0)
        x.copy_(torch.randn_like(x))
        K.MatVec(want, 1.0, x, 0.0)
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
