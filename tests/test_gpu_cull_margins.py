"""Boxes of voxels are culled only where their projection is accurate: small
boxes a hand's breadth in front of long lenses, far from the world's origin,
where a coordinate's rounding moves a projection by many pixels, and depth with
sharp steps.  All tile shapes and the batch against the passes without depth
pyramids (bricks 4-8) and the CPU oracle, bit for bit."""
import numpy as np
import pytest

from cuphoto import TSDFVolume, TSDFVolumeConfig, _lib as L
from cuphoto.batch import BatchIntegrator

from helpers import dev_depth, oracle_run

pytestmark = pytest.mark.gpu

GRID, VOXEL, FRAMES = (152, 144, 144), 0.00125, 16


def case(seed, offset, mode, arith):
    rng = np.random.default_rng(seed)
    w, h, f = 640, 480, 1500.0
    size = np.array(GRID) * VOXEL
    # (compat mode compares depth with world z: that stays near 0)
    off = np.array([offset, -0.7 * offset, 0.05 if mode == "compat" else 0.6 * offset])
    tc = TSDFVolumeConfig(voxel_grid_size=GRID, physical_size=tuple(size), global_offset=tuple(off), focal_x=f,
                          focal_y=f, cx=319.5, cy=239.5, mode=mode, arith=arith)
    depths, poses = [], []
    for _ in range(FRAMES):
        b = 2 ** rng.integers(3, 8)
        blocks = rng.choice([0, 0, 60, 120, 300, 2000], size=(h // b + 1, w // b + 1))
        d = np.roll(np.kron(blocks, np.ones((b, b), int)), rng.integers(0, 8, 2), (0, 1))[:h, :w]
        depths.append(np.ascontiguousarray(d.astype(np.uint16)))
        q = rng.normal(size=4)
        q /= np.linalg.norm(q)
        qw, x, y, z = q
        R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - qw * z), 2 * (x * z + qw * y)],
                      [2 * (x * y + qw * z), 1 - 2 * (x * x + z * z), 2 * (y * z - qw * x)],
                      [2 * (x * z - qw * y), 2 * (y * z + qw * x), 1 - 2 * (x * x + y * y)]])
        # a point of the volume on the axis of view, in front of the camera
        c = off + size * rng.uniform(0, 1, 3) - R[2] * rng.uniform(0.1, 0.35)
        poses.append(np.concatenate([q, -R @ c]))
    return tc, depths, np.array(poses)


@pytest.mark.parametrize("offset", [0.0, 3e3, 1e4, 3e4])
@pytest.mark.parametrize("mode,arith", [("compat", "ieee"), ("fixed", "ieee"), ("compat", "reference")])
def test_far_from_the_origin(gpu, oracle, mode, arith, offset):
    for seed in range(4):
        tc, depths, poses = case(seed, offset, mode, arith)
        dd = [dev_depth(gpu, d) for d in depths]

        def bits(brick, batch=False):
            vol = TSDFVolume(tc)
            built = L.debug_count(L.COUNT_PYRAMID_FRAMES)
            if batch:
                BatchIntegrator(1, FRAMES).integrate([vol], [dd], [poses], brick=brick)
            else:
                vol.integrate_frames(dd, poses, brick=brick)
            gpu.cuda.synchronize()
            assert L.debug_count(L.COUNT_PYRAMID_FRAMES) - built == (FRAMES if brick < 4 else 0)
            return (vol.voxel_distances_data().cpu().numpy().view(np.uint32).copy(),
                    vol.voxel_weights_data().cpu().numpy().copy())

        D0, W0 = bits(4)
        assert (W0 > 0).mean() > 0.1
        if arith == "ieee":
            Do, Wo = oracle_run(oracle, tc, depths, poses)
            assert np.array_equal(W0, Wo.reshape(W0.shape)) and np.array_equal(D0, Do.view(np.uint32).reshape(D0.shape))
        for brick, batch in [(0, False), (1, False), (2, False), (3, False), (5, False), (8, False), (0, True), (3, True)]:
            D, W = bits(brick, batch)
            assert np.array_equal(W, W0) and np.array_equal(D, D0), (seed, brick, batch)
