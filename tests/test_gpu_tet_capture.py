"""The tet assemblers allocate nothing after the mesh is made, whatever is assembled first: they can be captured into a
CUDA graph at once, and a graph stays valid when another form (stiffness warping, with its larger per-tet workspace) is
assembled on the same mesh afterwards. Replays give the bits of the call."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forms(torch, mesh, n):
    gen = torch.Generator(device="cuda").manual_seed(3)
    u, v, a = (0.01 * torch.randn(3 * n, dtype=torch.float64, device="cuda", generator=gen) for _ in range(3))
    E = 1.0 + torch.rand(mesh.ntet, dtype=torch.float64, device="cuda", generator=gen)
    rot = torch.eye(3, dtype=torch.float64, device="cuda").repeat(n, 1, 1).contiguous().reshape(-1)
    g = (0.0, 0.0, -1.0)
    return {
        "linear": lambda b: mesh.assemble_linear(E, 0.3, 1.0, g, b, u),
        "beuler": lambda b: mesh.assemble_beuler(1.0, 2.0, 1.5, g, 0.01, u, v, b),
        "newmark": lambda b: mesh.assemble_newmark(1.0, 2.0, 1.5, g, 0.01, 0.6, 0.36, u, v, a, b),
        "warp": lambda b: mesh.assemble_beuler(1.0, 2.0, 1.5, g, 0.01, u, v, b, rot),
    }


@pytest.mark.parametrize("form", ["linear", "beuler", "newmark", "warp"])
def test_assembly_is_captured(gpu, form):
    torch = pytest.importorskip("torch")
    import delfem2_gb300 as D
    from delfem2_gb300 import _native as N
    a = D.voxel_problem_arrays(5, 4, 6, 0.25, seed=1)
    n = a["np"]
    K = D.CMatrixSparse()
    K.Initialize(n, 3, True)
    K.SetPattern(a["psup_ind"], a["psup"])
    mesh = D.TetMesh(K, a["xyz"], a["tet"])
    forms = _forms(torch, mesh, n)
    b = torch.zeros(3 * n, dtype=torch.float64, device="cuda")

    def allocations():
        c = C.c_ulonglong(0)
        assert gpu.dfm2g_alloc_count(C.byref(c)) == N.OK
        return c.value

    before = allocations()
    K.setZero()
    forms[form](b)
    want = b.clone(), torch.from_numpy(K.get_values()[0])
    assert allocations() == before
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        forms[form](b)
    for other in forms.values():
        other(torch.zeros_like(b))
    b.zero_()
    K.setZero()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(b, want[0]) and torch.equal(torch.from_numpy(K.get_values()[0]), want[1])
    assert allocations() == before
