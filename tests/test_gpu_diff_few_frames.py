"""The differentiable forward and adjoint of so few frames that they are applied
without testing them against the boxes of voxels, beside those that are tested."""
import numpy as np
import pytest

from cuphoto.diff import backward_raw, forward_raw

from test_gpu_diff_cull import case, test_culled_equals_unculled as culled_equals_unculled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 2, 3, 4])
@pytest.mark.parametrize("grid", [(33, 13, 5), (23, 30, 17)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_forward_equals_the_one_that_tests_nothing(gpu, grid, frames, dtype):
    culled_equals_unculled(gpu, grid, frames, 0.05, dtype)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_adjoint_with_and_without_tests(gpu, dtype):
    """Three frames alone and with a fourth that holds no depth: one voxel, whose
    gradients are no sums, so they are equal bit for bit."""
    dt = getattr(gpu, dtype)
    seen = 0
    for seed in range(200):
        cfg, R, t, depth = case((1, 1, 1), 4, seed, 0.05)
        depth[3] = 0.0
        outs = []
        for n in (3, 4):
            Rn, tn, dn = (gpu.tensor(a[:n], dtype=dt, device="cuda") for a in (R, t, depth))
            D0 = gpu.full((1, 1, 1), cfg.truncation, dtype=dt, device="cuda")
            W0 = gpu.zeros((1, 1, 1), dtype=dt, device="cuda")
            D, W = D0.clone(), W0.clone()
            forward_raw(cfg, D, W, dn, Rn, tn)
            gD, gW = gpu.full_like(D0, 1.3), gpu.full_like(D0, -0.7)
            gdep, gpose = gpu.zeros_like(dn), gpu.zeros((n, 12), dtype=gpu.float64, device="cuda")
            gD0, gW0 = gpu.empty_like(D0), gpu.empty_like(W0)
            backward_raw(cfg, gD, gW, D0, W0, None, dn, Rn, tn, gdep, gpose, gD0, gW0)
            outs.append([x.cpu().numpy() for x in (D, W, gdep[:3], gpose[:3], gD0, gW0)])
        for a, b in zip(*outs):
            assert np.array_equal(a, b)
        seen += bool(outs[0][1].any())
    assert seen > 20
