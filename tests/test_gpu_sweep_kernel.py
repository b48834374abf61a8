"""Which kernel a sweep ran (dfm2g_ilu_last_kernel): the one over tiles wherever the pattern's rows fit its records (at
most 15 blocks in a triangle: 7 for voxel meshes, 13 for ILU(1) of them, 27 and more for ILU(2)) and the partition
averages at least 16 rows a tile, a warp per chain otherwise, for the automatic choice and DFM2G_SWEEP_CHAINS, every
block size, precision and direction; the rows per tile come from dfm2g_tile_partition with the sweeps' tile sizes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SYNCFREE, LEVELS, CHAINS, TILES, AUTO = 0, 1, 5, 6, 7


def _handle(dims, ndim, fill=0, perm=False, cloth=0):
    import delfem2_gb300 as D
    from delfem2_gb300 import cloth as DC
    if cloth:
        n = (cloth + 1) ** 2
        ind, psup = D.JArray_PSuP_MeshElem(DC.SetClothShape_Square(cloth, 1.0)[3], 4, n)
    else:
        xyz, tet = D.MeshTet3D_VoxelGrid(*dims, 1.0)
        n = xyz.size // 3
        if perm:
            tet = np.random.default_rng(7).permutation(n).astype(np.uint32)[tet]
        ind, psup = D.JArray_PSuP_MeshElem(tet, 4, n)
    rng = np.random.default_rng(n)
    K = D.CMatrixSparse()
    K.Initialize(n, ndim, True)
    K.SetPattern(ind, psup)
    K.set_values(0.02 * rng.standard_normal(np.asarray(psup).size * ndim * ndim), np.tile(np.eye(ndim).ravel(), n))
    ilu = D.CPreconditionerILU()
    ilu.Initialize_ILUk(K, fill)
    ilu.CopyValue(K)
    assert ilu.Decompose()
    return ilu, n * ndim


def _rule(lib, ilu, ndim, fp64):
    rs = np.ascontiguousarray(ilu.row_start(), np.uint32)
    col, dia = (np.ascontiguousarray(a, np.uint32) for a in ilu.pattern())
    n, segs = rs.size - 1, {1: 64, 2: 32, 3: 16 if fp64 else 36}[ndim]
    out = []
    for backward in (False, True):
        order = np.ascontiguousarray(ilu.levels(backward)[1], np.uint32)
        tile_of, level = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
        nt, m = C.c_uint(0), C.c_uint(0)
        assert lib.dfm2g_tile_partition(n, rs.ctypes.data, col.ctypes.data, dia.ctypes.data, order.ctypes.data,
                                        int(backward), 65 * segs, segs, tile_of.ctypes.data, level.ctypes.data,
                                        C.byref(nt), C.byref(m)) == 0
        out.append(TILES if m.value <= 15 and (nt.value == 1 or n >= 16 * nt.value) else CHAINS)
    return out


@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("kw,want", [
    (dict(dims=(12, 11, 13)), TILES), (dict(dims=(3, 2, 2)), TILES), (dict(dims=(), cloth=30), TILES),
    (dict(dims=(9, 8, 10), fill=1), TILES), (dict(dims=(9, 8, 10), fill=2), CHAINS),
    (dict(dims=(14, 13, 12), perm=True), CHAINS)])
def test_kernel_of_the_sweep(gpu, ndim, kw, want):
    ilu, n = _handle(ndim=ndim, **kw)
    assert [ilu.last_kernel(f, b) for f in (False, True) for b in (False, True)] == [-1] * 4
    for mode in (AUTO, CHAINS):
        ilu.set_sweep_mode(mode)
        for fp64, dtype in ((True, np.float64), (False, np.float32)):
            assert _rule(gpu, ilu, ndim, fp64) == [want, want]
            ilu.SolvePrecond(np.ones(n, dtype))
            assert [ilu.last_kernel(fp64, b) for b in (False, True)] == [want, want], (mode, fp64)
    for mode in (SYNCFREE, LEVELS):
        ilu.set_sweep_mode(mode)
        ilu.SolvePrecond(np.ones(n))
        assert [ilu.last_kernel(True, b) for b in (False, True)] == [mode, mode]
        assert [ilu.last_schedule(True, b) for b in (False, True)] == [mode, mode]


def test_last_kernel_rejects_bad_arguments(gpu):
    from delfem2_gb300 import _native as N
    ilu, _ = _handle((3, 2, 2), 3)
    m = C.c_int(0)
    assert gpu.dfm2g_ilu_last_kernel(ilu._h, 5, 0, C.byref(m)) != 0
    assert gpu.dfm2g_ilu_last_kernel(ilu._h, N.F32, 0, None) != 0
    assert gpu.dfm2g_ilu_last_kernel(None, N.F32, 0, C.byref(m)) != 0


@pytest.mark.parametrize("modes", [(TILES, AUTO), (AUTO, TILES, AUTO), (TILES, CHAINS, TILES)])
def test_a_forced_schedule_is_not_taken_unasked(gpu, modes):
    """Thin tiles, once built for DFM2G_SWEEP_TILES, stay off the other modes' sweeps; the results agree."""
    ilu, n = _handle((14, 13, 12), 3, perm=True)
    b = np.random.default_rng(1).standard_normal(n)
    first = None
    for mode in modes:
        ilu.set_sweep_mode(mode)
        for fp64, dtype in ((True, np.float64), (False, np.float32)):
            x = b.astype(dtype)
            ilu.SolvePrecond(x)
            want = TILES if mode == TILES else CHAINS
            assert [ilu.last_kernel(fp64, k) for k in (False, True)] == [want, want], (mode, fp64)
            if first is None:
                first = x
            assert np.abs(x - first).max() < (1e-12 if fp64 else 1e-5) * np.abs(first).max()
