"""Lanes per node of the tet assembly (csrc/fem.cu: 8, 4 or 2 as long as the mesh's lanes stay within a warp for each SM
quarter, else 1) on both sides of each change: voxel blocks of 2,420 / 2,448, 4,851 / 4,896 and 9,702 / 9,747 nodes (152
SMs: 2,432, 4,864 and 9,728), against the oracle. Static elasticity with a displacement, the stiffness-warped step and
the Newmark form. Tolerance 1e-12 relative (sums of at most 24 tets, each rounded to 1.1e-16, over entries of one
magnitude)."""
import numpy as np
import pytest

from conftest import rel_err
from dyn_systems import MAT, rotations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(10, 10, 19), (11, 11, 16), (10, 20, 20), (11, 16, 23), (20, 20, 21), (18, 18, 26)])
def test_lane_counts(gpu, port, dims):
    import delfem2_gb300 as D
    xyz, tet = port.voxel_tet_mesh(*dims, 0.3)
    npn, ntet = xyz.size // 3, tet.size // 4
    ind, psup = (np.asarray(a, np.uint32) for a in port.psup(tet, 4, npn))
    rng = np.random.default_rng(6)
    E, u, v, acc = rng.uniform(0.1, 10, ntet), *(rng.standard_normal((3, npn * 3)))
    rot, m = rotations(npn), MAT
    for kind in ("linear", "warp", "newmark"):
        K = D.CMatrixSparse()
        K.Initialize(npn, 3, True)
        K.SetPattern(ind, psup)
        K.setZero()
        mesh, b = D.TetMesh(K, xyz, tet), np.zeros(npn * 3)
        if kind == "linear":
            mesh.assemble_linear(E, 0.3, 1.5, (0.1, 0.2, -9.8), b, u)
            want = np.zeros(psup.size * 9), np.zeros(npn * 9), np.zeros(npn * 3)
            assert port.assemble_tet_linear(ind, psup, *want, xyz, tet, E, 0.3, 1.5, [0.1, 0.2, -9.8], u) == 0
        elif kind == "warp":
            mesh.assemble_beuler(m["myu"], m["lam"], m["rho"], m["g"], m["dt"], u, v, b, rot)
            want = port.assemble_tet_beuler(ind, psup, xyz, tet, m["myu"], m["lam"], m["rho"], m["g"], m["dt"], u, v,
                                            rot)
        else:
            mesh.assemble_newmark(m["myu"], m["lam"], m["rho"], m["g"], m["dt"], m["gamma"], m["beta"], u, v, acc, b)
            want = port.assemble_tet_newmark(ind, psup, xyz, tet, m["myu"], m["lam"], m["rho"], m["g"], m["dt"],
                                             m["gamma"], m["beta"], u, v, acc)
        gc, gd = K.get_values()
        assert rel_err(gc, want[0]) < 1e-12 and rel_err(gd, want[1]) < 1e-12 and rel_err(b, want[2]) < 1e-12
