"""Tile sweeps (DFM2G_SWEEP_TILES / DFM2G_SWEEP_CHAINS, csrc/tile_kernel.cuh) at the sizes where their layout
turns over, against the oracle: z lines of 65 and 66 rows (one segment, two), grids of one line more than a tile's
square (4 x 4 lines in FP64, 6 x 6 in FP32), a single row, more than one tile per CTA, lane groups of 1x1, 2x2 and
3x3 blocks, ILU(1) rows (13 dependencies: the long-row kernels), and rows numbered at random, whose tiles of about
ten rows are swept only when the tile schedule is asked for. Tolerances: 1e-12 relative in FP64 (summation order
only; the condition of these systems is below 1e2), 1e-5 in FP32 (some 20 roundings of 6e-8 along at most 80 levels
of a contracting recurrence)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TILES, CHAINS, AUTO = 6, 5, 7


def _grid_pattern(port, nx, ny, nz, perm=False):
    """The adjacency of a voxel block of nx x ny x nz nodes (six tets a cell)."""
    if min(nx, ny, nz) < 2:  # a line or a single row: tridiagonal
        n = nx * ny * nz
        nbr = [[j for j in (i - 1, i + 1) if 0 <= j < n] for i in range(n)]
        ind = np.concatenate([[0], np.cumsum([len(a) for a in nbr])]).astype(np.uint32)
        return ind, np.array([j for a in nbr for j in a], np.uint32)
    xyz, tet = port.voxel_tet_mesh(nx - 1, ny - 1, nz - 1, 1.0)
    n = xyz.size // 3
    if perm:
        tet = np.random.default_rng(7).permutation(n).astype(np.uint32)[tet]
    ind, psup = port.psup(tet, 4, n)
    return np.asarray(ind, np.uint32), np.asarray(psup, np.uint32)


def _sweeps(port, dims, ndim, fill=0, perm=False):
    import delfem2_gb300 as D
    ind, psup = _grid_pattern(port, *dims, perm)
    n, bb = ind.size - 1, ndim * ndim
    rng = np.random.default_rng(n + ndim)
    vc = 0.2 / ndim * rng.standard_normal(psup.size * bb)
    vd = np.tile(np.eye(ndim).ravel(), n) * 4.0 + 0.1 * rng.standard_normal(n * bb)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(vc, vd)
    ilu = D.CPreconditionerILU()
    ilu.Initialize_ILUk(K, fill)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    rs = np.asarray(ilu.row_start())
    col, dia = ilu.pattern()
    return ilu, n * ndim, (ndim, rs, col, dia) + tuple(ilu.values())


def _check(port, ilu, n, o):
    nd, rs, col, dia, vc, vd = o
    v = np.random.default_rng(3).standard_normal(n)
    if nd == 3:
        fo = port.ilu_forward(rs, col, dia, vc, vd, v)
        go = port.ilu_backward(rs, col, dia, vc, fo)
    else:
        fo = port.nd_ilu_forward(nd, rs, col, dia, vc, vd, v)
        go = port.nd_ilu_backward(nd, rs, col, dia, vc, fo)
    f, g, z = v.copy(), fo.copy(), v.astype(np.float32)
    ilu.ForwardSubstitution(f)
    ilu.BackwardSubstitution(g)
    ilu.SolvePrecond(z)
    assert rel_err(f, fo) < 1e-12 and rel_err(g, go) < 1e-12 and rel_err(z, go) < 1e-5


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 1, 66), (2, 2, 2), (4, 4, 65), (5, 4, 66), (7, 6, 3), (13, 9, 11)])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_tile_edges(gpu, port, dims, ndim):
    ilu, n, o = _sweeps(port, dims, ndim)
    _check(port, ilu, n, o)
    if ndim == 3:
        ilu.set_sweep_mode(TILES)
        _check(port, ilu, n, o)
        assert ilu.last_schedule(True, False) == TILES


def test_long_rows_and_many_tiles(gpu, port):
    _check(port, *_sweeps(port, (9, 8, 10), 3, fill=1))
    _check(port, *_sweeps(port, (60, 59, 7), 3))  # about 225 FP64 tiles: more than the SMs


def test_random_numbering(gpu, port):
    ilu, n, o = _sweeps(port, (14, 13, 12), 3, perm=True)
    _check(port, ilu, n, o)
    assert ilu.last_schedule(True, False) == CHAINS
    ilu.set_sweep_mode(TILES)  # asked for: thin tiles are built and swept
    _check(port, ilu, n, o)
    assert ilu.last_schedule(True, False) == TILES
