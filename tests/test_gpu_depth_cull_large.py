"""The checks of test_gpu_depth_cull and test_gpu_odd_states on grids so large that
16-frame passes build depth pyramids (49 M voxel-frames; their line lies at 42 M for
frames of 320x240), in every tile shape and the batch."""
import numpy as np
import pytest

from cuphoto import TSDFVolume, _lib as L
from cuphoto.batch import BatchIntegrator

import test_gpu_depth_cull as small
import test_gpu_odd_states as odd
from helpers import dev_depth, frontal_case, oracle_run

pytestmark = pytest.mark.gpu

GRIDS = [(152, 144, 144), (149, 143, 145)]


def pyramids(call):
    n = L.debug_count(L.COUNT_PYRAMID_FRAMES)
    call()
    return L.debug_count(L.COUNT_PYRAMID_FRAMES) - n


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("fmt", ["u16", "f32"])
@pytest.mark.parametrize("path", ["frontal", "circle"])
@pytest.mark.parametrize("mode,arith", [("compat", "ieee"), ("fixed", "ieee"), ("compat", "reference")])
def test_passes_and_batches(gpu, oracle, grid, fmt, path, mode, arith):
    built = pyramids(lambda: small.test_passes_and_batches_with_pyramids(gpu, oracle, grid, fmt, path, mode, arith))
    assert built == 4 * 16 + 4 * 16 + 32   # passes and batches of four tile shapes, a pass of 32 frames


def test_negative_scale_and_short_range(gpu, oracle):
    depths, poses, cam = small.frames("circle", "u16", 3)
    dd = [dev_depth(gpu, d) for d in depths]
    near = small.config("circle", GRIDS[0], cam, mode="fixed", max_depth=1.4)
    far = small.config("circle", GRIDS[0], cam, mode="fixed", max_depth=9.0)
    a, b = TSDFVolume(near), TSDFVolume(far)
    assert pyramids(lambda: BatchIntegrator(2, 32).integrate([a, b], [dd, dd], [poses, poses])) == 32
    for vol, tc in ((a, near), (b, far)):
        D, W = small.volume_bits(gpu, vol)
        Do, Wo = oracle_run(oracle, tc, depths, poses)
        assert np.array_equal(W, Wo.reshape(W.shape)) and np.array_equal(D, Do.view(np.uint32).reshape(D.shape))
    D0, W0 = small.volume_bits(gpu, a)
    assert pyramids(lambda: a.integrate_frames(dd, poses, depth_scale=-0.001)) == 16
    D, W = small.volume_bits(gpu, a)
    assert np.array_equal(W, W0) and np.array_equal(D, D0)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("mode", ["compat", "fixed"])
def test_odd_states(gpu, oracle, grid, mode):
    seq, tc = frontal_case(*grid, 16, mode=mode, arith="ieee")
    assert pyramids(lambda: odd.compare(gpu, oracle, tc, seq, 16, np.random.default_rng(grid[0]), True)) == 16
