"""IEEE integrate in both modes on states and poses where paired quotients and
reciprocals have to give way to plain ones, against the CPU oracle bit for bit: fractional, negative, huge,
infinite and NaN weights, tiny and huge distances, rotations from quaternions that
are not of unit length, cameras among the voxels."""
import numpy as np
import pytest

from cuphoto import TSDFVolume
from cuphoto import synthetic as S

from helpers import circle_case, dev_depth, frontal_case, set_distances

pytestmark = pytest.mark.gpu

WEIGHTS = np.array([0, 1, 5, 127, 300, 0.1, 2.7, -0.3, -1, -1.5, -7, 1e-30, 3e7, 1e20, np.inf, -np.inf, np.nan], np.float32)
DISTANCES = np.array([0, -0.0, 0.05, -0.03, 1e-12, -1e-26, 1e-38, 1e-42, 3e24, -1e36, 3e38, np.inf, np.nan], np.float32)


def compare(gpu, oracle, tc, seq, n, rng, odd):
    vol = TSDFVolume(tc)
    c = oracle.cfg_from(tc)
    D, W = oracle.init_volume(c)
    if odd:
        pick = rng.random(D.shape)
        weights = WEIGHTS if tc.mode == "compat" else WEIGHTS[~(WEIGHTS > 2e9)]   # (whole parts are 32-bit)
        W[:] = np.where(pick < 0.5, rng.integers(0, 200, D.shape), weights[rng.integers(0, len(weights), D.shape)])
        D[:] = np.where(pick < 0.7, rng.uniform(-0.1, 0.1, D.shape), DISTANCES[rng.integers(0, len(DISTANCES), D.shape)])
        set_distances(gpu, vol, D, W)
    before = W.copy()
    depths = [d.astype(np.float32) * np.float32(0.001) for d in seq.depth_u16[:n]]
    vol.integrate_frames([dev_depth(gpu, d) for d in depths], seq.poses[:n])
    for d, p in zip(depths, seq.poses[:n]):
        if tc.mode == "compat":
            oracle.integrate_compat(c, D, W, d, p)
        else:
            oracle.integrate_fixed(c, D, W, d, p, 0.001)
    gpu.cuda.synchronize()
    gD, gW = vol.voxel_distances_data().cpu().numpy().reshape(D.shape), vol.voxel_weights_data().cpu().numpy().reshape(D.shape)
    for got, want in ((gD, D), (gW, W)):
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])
    assert (W != before).any()


# one frame: voxels along x; three: along z; sixteen: with depth pyramids; rows of
# 93: single voxels at the edge
@pytest.mark.parametrize("frames", [1, 3, 16])
@pytest.mark.parametrize("nx", [96, 93])
@pytest.mark.parametrize("mode", ["compat", "fixed"])
def test_odd_states(gpu, oracle, frames, nx, mode):
    seq, tc = frontal_case(nx, 80, 72, frames, mode=mode, arith="ieee")
    compare(gpu, oracle, tc, seq, frames, np.random.default_rng(frames + nx), True)


@pytest.mark.parametrize("mode", ["compat", "fixed"])
@pytest.mark.parametrize("scale", [1.0, 1.7, 12.0])
@pytest.mark.parametrize("physical", [2.56, 0.02])
def test_odd_poses(gpu, oracle, mode, scale, physical):
    seq, tc = circle_case(96, 16, physical=physical, mode=mode, arith="ieee")
    if mode == "compat":   # (the fixed mode normalises)
        seq.poses[::2, :4] *= np.asarray(scale, seq.poses.dtype)
    seq.poses[1::4, 4:] *= np.asarray(0.02, seq.poses.dtype)   # among the voxels
    if physical < 1.0:
        seq.poses[:, 4:] *= np.asarray(0.01, seq.poses.dtype)
    compare(gpu, oracle, tc, seq, 16, np.random.default_rng(1), False)
