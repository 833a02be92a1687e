"""One frame per call into grids from 12 M voxels on, whose threads hold voxels along
x (rows of a multiple of 4; IEEE arithmetic's and the others') and which build a
depth pyramid for the frame: against the passes without pyramids and the CPU
oracle, bit for bit, on frames with holes, without depth, with unusable values,
and of odd sizes."""
import numpy as np
import pytest

from cuphoto import TSDFVolume, _lib as L

from helpers import dev_depth, oracle_run
from test_gpu_depth_cull import config, frames, volume_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(240, 232, 236), (236, 233, 239), (237, 232, 240)])
@pytest.mark.parametrize("path,fmt", [("frontal", "u16"), ("circle", "f32")])
@pytest.mark.parametrize("mode,arith", [("compat", "ieee"), ("fixed", "ieee"), ("compat", "reference")])
def test_single_frames(gpu, oracle, grid, path, fmt, mode, arith):
    assert np.prod(grid) >= 12 << 20
    depths, poses, cam = frames(path, fmt, 6, n=9)
    tc = config(path, grid, cam, mode=mode, arith=arith)
    dd = [dev_depth(gpu, d) for d in depths]
    plain = TSDFVolume(tc)
    for d, p in zip(dd, poses):
        plain.integrate_frames([d], [p], brick=4)     # depth staged in shared memory: no pyramids
    D0, W0 = volume_bits(gpu, plain)
    assert (W0 > 0).any() and (W0 == 0).any()
    vol = TSDFVolume(tc)
    for brick in range(4):
        vol.reset()
        built = L.debug_count(L.COUNT_PYRAMID_FRAMES)
        for d, p in zip(dd, poses):
            if brick == 0:
                assert vol.integrate(d, d, p)
            else:
                vol.integrate_frames([d], [p], brick=brick)
        assert L.debug_count(L.COUNT_PYRAMID_FRAMES) - built == len(dd)
        D, W = volume_bits(gpu, vol)
        assert np.array_equal(W, W0) and np.array_equal(D, D0), brick
    if arith == "ieee":
        Do, Wo = oracle_run(oracle, tc, depths, poses)
        assert np.array_equal(W0, Wo.reshape(W0.shape)) and np.array_equal(D0, Do.view(np.uint32).reshape(D0.shape))
