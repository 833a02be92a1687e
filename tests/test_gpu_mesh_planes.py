"""The mesh counted and emitted from bit planes, where its words, quarters and
sixteenths of tiles and runs of rows end, against the CPU oracle bit for bit:
the tolerance of the other mesh tests."""
import numpy as np
import pytest

from cuphoto import TSDFVolume, TSDFVolumeConfig, extract_mesh_indexed

from helpers import mesh, set_distances

pytestmark = pytest.mark.gpu

GRIDS = [(2, 2, 2), (33, 2, 3), (32, 34, 3), (34, 5, 4), (65, 9, 7), (31, 33, 35), (513, 6, 5), (3, 700, 4), (8, 3, 600),
         (130, 70, 9)]


def field(kind, grid, seed):
    """Distances and weights (z, y, x): signs at random (tiles full of
    triangles), one voxel below zero, or a flat surface along x."""
    rng = np.random.default_rng(seed)
    shape = grid[::-1]
    W = np.ones(shape, np.float32)
    if kind == "noise":
        D = rng.normal(size=shape).astype(np.float32)
        D.reshape(-1)[::97] = 0.0
        D.reshape(-1)[5::101] = -0.0
        W[rng.random(shape) < 0.03] = 0
    elif kind == "one":
        D = np.full(shape, 0.3, np.float32)
        D[tuple(s // 2 for s in shape)] = -0.2
    else:
        D = np.broadcast_to((np.arange(shape[1])[None, :, None] - 0.4 * shape[1]), shape).astype(np.float32).copy()
        W[..., -1] = 0
    return D, W


@pytest.mark.parametrize("kind", ["noise", "one", "flat"])
@pytest.mark.parametrize("grid", GRIDS)
def test_fixed_mesh(gpu, oracle, grid, kind):
    tc = TSDFVolumeConfig(voxel_grid_size=grid, physical_size=tuple(0.01 * g for g in grid),
                          global_offset=(-0.3, 0.2, 0.5), mode="fixed", max_weight=16)
    vol = TSDFVolume(tc)
    D, W = field(kind, grid, sum(grid))
    set_distances(gpu, vol, D, W)
    V, T = mesh(vol)
    Vo, To = oracle.mc_fixed(oracle.cfg_from(tc), D.ravel(), W.ravel())
    assert len(V) == len(Vo) and np.array_equal(T, To)
    assert np.array_equal(V.view(np.uint32), Vo.view(np.uint32))
    Vi, _, Ti = (x.cpu().numpy() for x in extract_mesh_indexed(vol))
    assert len(Ti) == len(T) and np.unique(Ti).size == len(Vi)
    assert np.array_equal(Vi[Ti].view(np.uint32), V.view(np.uint32))


@pytest.mark.parametrize("kind", ["noise", "one", "flat"])
@pytest.mark.parametrize("grid", GRIDS)
def test_compat_mesh(gpu, oracle, grid, kind):
    tc = TSDFVolumeConfig(voxel_grid_size=grid, physical_size=tuple(0.01 * g for g in grid),
                          global_offset=(-0.3, 0.2, 0.5), arith="ieee")
    vol = TSDFVolume(tc)
    D, _ = field(kind, grid, 3 + sum(grid))
    set_distances(gpu, vol, D)
    V, T = mesh(vol)
    Vo, To = oracle.mc_compat(oracle.cfg_from(tc), D.ravel())
    assert len(V) == len(Vo) and np.array_equal(T, To)
    assert np.array_equal(V.view(np.uint32), Vo.view(np.uint32))


def test_sized_extraction_counts_once_and_reports(gpu):
    """gbt_extract_mesh_sized: the counts given to alloc, a refusing alloc, an
    index range that does not fit (before alloc), shared vertices in compat."""
    import ctypes as C
    from cuphoto import _lib as L
    lib = L.lib()
    grid = (40, 36, 32)
    size = dict(voxel_grid_size=grid, physical_size=tuple(0.01 * g for g in grid))
    vol = TSDFVolume(TSDFVolumeConfig(mode="fixed", max_weight=16, **size))
    D, W = field("noise", grid, 5)
    set_distances(gpu, vol, D, W)
    V, T = mesh(vol)
    seen = []

    def refuse(ctx, nv, nt, v, n, t):
        seen.append((nv, nt))
        return 1

    cb = L.MESH_ALLOC(refuse)
    nv, nt = C.c_int64(-1), C.c_int64(-1)
    args = (cb, None)
    assert lib.gbt_extract_mesh_sized(vol.handle, 0, *args, 0, C.byref(nv), C.byref(nt), None) == L.GBT_ERR_ALLOC
    assert seen == [(3 * len(T), len(T))] and (nv.value, nt.value) == (0, 0)
    assert lib.gbt_extract_mesh_sized(vol.handle, 1, *args, 0, C.byref(nv), C.byref(nt), None) == L.GBT_ERR_ALLOC
    assert seen[1][1] == len(T) and 0 < seen[1][0] < 3 * len(T)
    base = 2 ** 31 - 10
    assert lib.gbt_extract_mesh_sized(vol.handle, 0, *args, base, C.byref(nv), C.byref(nt), None) == L.GBT_ERR_INVALID_ARG
    compat = TSDFVolume(TSDFVolumeConfig(**size))
    assert lib.gbt_extract_mesh_sized(compat.handle, 1, *args, 0, C.byref(nv), C.byref(nt), None) == L.GBT_ERR_INVALID_ARG
    assert len(seen) == 2
    V2, T2 = mesh(vol)
    assert np.array_equal(V2.view(np.uint32), V.view(np.uint32)) and np.array_equal(T2, T)
