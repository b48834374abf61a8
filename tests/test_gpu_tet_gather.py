"""The gathered tet assembly (csrc/fem.cu) on meshes whose gather lists are uneven, against the oracle: a fan of tets
around one edge (an edge and two nodes in every tet, more than a warp's worth), a single tet, tets in reversed and
shuffled order, and nodes no tet touches. Static elasticity with a displacement, the stiffness-warped step, the
Newmark form and the scalar problem. Tolerance 1e-12 relative (sums of at most some 300 terms, each rounded to
1.1e-16, over entries of one magnitude)."""
import numpy as np
import pytest

from conftest import rel_err
from dyn_systems import MAT, rotations

pytestmark = pytest.mark.gpu


def _fan(n, shuffle):
    """n tets around the edge (0, 1), closed ring; two more nodes belong to no tet."""
    th = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(th), np.sin(th), 0.1 * np.cos(3 * th)], 1)
    xyz = np.concatenate([[[0, 0, -1.0], [0, 0, 1.2]], ring, [[5.0, 5, 5], [6, 5, 5]]])
    k = np.arange(n)
    tet = np.stack([0 * k, 2 + k, 2 + (k + 1) % n, 0 * k + 1], 1).astype(np.uint32)
    if shuffle:
        tet = tet[np.random.default_rng(n).permutation(n)]
    return xyz.ravel(), tet.ravel()


def _single():
    return np.array([0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1.0]), np.arange(4, dtype=np.uint32)


@pytest.mark.parametrize("n,shuffle", [(1, False), (3, False), (33, True), (140, True)])
def test_uneven_lists(gpu, port, n, shuffle):
    import delfem2_gb300 as D
    xyz, tet = _single() if n == 1 else _fan(n, shuffle)
    npn, ntet = xyz.size // 3, tet.size // 4
    ind, psup = port.psup(tet, 4, npn)
    ind, psup = np.asarray(ind, np.uint32), np.asarray(psup, np.uint32)
    rng = np.random.default_rng(5)
    E, u, v, acc = rng.uniform(0.1, 10, ntet), *(rng.standard_normal((3, npn * 3)))
    rot, val = rotations(npn), rng.standard_normal(npn)

    def fresh(ndim):
        K = D.CMatrixSparse()
        K.Initialize(npn, ndim, True)
        K.SetPattern(ind, psup)
        K.setZero()
        return K, D.TetMesh(K, xyz, tet), np.zeros(npn * ndim)

    def check(K, b, want):
        vc, vd, bo = want
        gc, gd = K.get_values()
        assert rel_err(gc, vc) < 1e-12 and rel_err(gd, vd) < 1e-12 and rel_err(b, bo) < 1e-12

    K, mesh, b = fresh(3)
    mesh.assemble_linear(E, 0.3, 1.5, (0.1, 0.2, -9.8), b, u)
    vc, vd, bo = np.zeros(psup.size * 9), np.zeros(npn * 9), np.zeros(npn * 3)
    assert port.assemble_tet_linear(ind, psup, vc, vd, bo, xyz, tet, E, 0.3, 1.5, [0.1, 0.2, -9.8], u) == 0
    check(K, b, (vc, vd, bo))
    m = MAT
    for kind in ("beuler", "warp", "newmark"):
        K, mesh, b = fresh(3)
        if kind == "newmark":
            mesh.assemble_newmark(m["myu"], m["lam"], m["rho"], m["g"], m["dt"], m["gamma"], m["beta"], u, v, acc, b)
            want = port.assemble_tet_newmark(ind, psup, xyz, tet, m["myu"], m["lam"], m["rho"], m["g"], m["dt"],
                                             m["gamma"], m["beta"], u, v, acc)
        else:
            r = rot if kind == "warp" else None
            mesh.assemble_beuler(m["myu"], m["lam"], m["rho"], m["g"], m["dt"], u, v, b, r)
            want = port.assemble_tet_beuler(ind, psup, xyz, tet, m["myu"], m["lam"], m["rho"], m["g"], m["dt"], u, v,
                                            r)
        check(K, b, want)
    K, mesh, b = fresh(1)
    mesh.assemble_poisson(0.7, 1.3, b, val)
    check(K, b, port.assemble_poisson_tet(ind, psup, xyz, tet, 0.7, 1.3, val))
