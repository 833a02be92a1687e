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
