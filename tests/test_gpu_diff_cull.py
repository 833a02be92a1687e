"""The differentiable forward and adjoint with frames culled per box of 8 x 4
voxels, against the forward that records every decision (it culls nothing) and
against the oracle: extents around the boxes, cameras inside the volume, behind
it, turned away and with min_z at and below 0; more frames than a warp has
lanes."""
import numpy as np
import pytest

from cuphoto import synthetic as S
from cuphoto.diff import DiffConfig, backward_raw, checkpoint_shape, forward_raw

pytestmark = pytest.mark.gpu


def case(grid, frames, seed, min_z):
    rng = np.random.default_rng(seed)
    cam = S.Camera(64, 48, 50.0, 50.0, 31.5, 23.5)
    R, t, depth = [], [], []
    for k in range(frames):
        c = rng.uniform(-1.6, 1.6, 3)                       # inside, near and around the volume
        target = rng.uniform(-1.0, 1.0, 3) if k % 3 else c + rng.normal(size=3)
        Rk, tk = S.look_at(c, target)
        R.append(Rk)
        t.append(tk)
        d = rng.uniform(0.2, 2.5, (cam.height, cam.width))
        d[rng.random(d.shape) < 0.2] = 0
        depth.append(d)
    vs = tuple(2.0 / g for g in grid)
    cfg = DiffConfig(grid, vs, (-1.0, -1.0, -1.0), cam.fx, cam.fy, cam.cx, cam.cy, 0.25, max_weight=6.0, max_depth=4.0,
                     min_z=min_z)
    return cfg, np.stack(R), np.stack(t), np.stack(depth)


@pytest.mark.parametrize("grid,frames", [((1, 1, 1), 3), ((7, 3, 2), 5), ((8, 4, 3), 9), ((33, 13, 5), 35), ((24, 30, 17), 70)])
@pytest.mark.parametrize("min_z", [0.05, 0.0, -0.5])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_culled_equals_unculled(gpu, grid, frames, min_z, dtype):
    cfg, R, t, depth = case(grid, frames, sum(grid) + frames, min_z)
    dt = getattr(gpu, dtype)
    R, t, depth = (gpu.tensor(a, dtype=dt, device="cuda") for a in (R, t, depth))
    shape = grid[::-1]
    outs = []
    for signed in (False, True):
        D = gpu.full(shape, cfg.truncation, dtype=dt, device="cuda")
        W = gpu.zeros(shape, dtype=dt, device="cuda")
        ck = gpu.zeros(checkpoint_shape(frames, shape), dtype=dt, device="cuda")
        sig = gpu.zeros(shape, dtype=gpu.int32, device="cuda") if signed else None
        forward_raw(cfg, D, W, depth, R, t, ck if ck.numel() else None, sig)
        outs.append((D, W, ck))
    gpu.cuda.synchronize()
    for a, b in zip(*outs):
        assert gpu.equal(a, b)
    D, W, ck = outs[0]
    if grid == (24, 30, 17):
        assert (W > 0).any() and (W == 0).any()
    # the adjoint's gradient to D0: each voxel's D is affine in its D0
    D0 = gpu.full(shape, cfg.truncation, dtype=dt, device="cuda")
    W0 = gpu.zeros(shape, dtype=dt, device="cuda")
    gD = gpu.ones(shape, dtype=dt, device="cuda")
    gdep, gpose = gpu.zeros_like(depth), gpu.zeros((frames, 12), dtype=gpu.float64, device="cuda")
    gD0, gW0 = gpu.empty_like(D0), gpu.empty_like(W0)
    backward_raw(cfg, gD, None, D0, W0, ck if ck.numel() else None, depth, R, t, gdep, gpose, gD0, gW0)
    D1 = D0 + 0.5
    W1 = W0.clone()
    forward_raw(cfg, D1, W1, depth, R, t)
    # (D1 - D) / 0.5: rounding of D (at most 1 in size) over 0.5, a few of them
    eps = float(gpu.finfo(dt).eps)
    assert float((gD0 - (D1 - D) / 0.5).abs().max()) <= 16 * eps * (1 + frames)


def test_adjoint_against_the_oracle(gpu, oracle):
    cfg, R, t, depth = case((17, 13, 9), 37, 3, 0.05)
    c = oracle.diff_cfg((17, 13, 9), cfg.voxel_size, cfg.global_offset, (cfg.focal_x, cfg.focal_y, cfg.cx, cfg.cy),
                        cfg.truncation, cfg.max_weight, cfg.max_depth, cfg.min_z, 64, 48, 1)
    shape = (9, 13, 17)
    rng = np.random.default_rng(1)
    gD, gW = rng.normal(size=shape), rng.normal(size=shape)
    Do, Wo = np.full(shape, cfg.truncation), np.zeros(shape)
    want = oracle.diff_backward(c, gD, gW, Do, Wo, depth, R, t)
    dev = [gpu.tensor(a, dtype=gpu.float64, device="cuda") for a in (gD, gW, Do, Wo, depth, R, t)]
    gD_, gW_, D0, W0, dep, R_, t_ = dev
    D, W = D0.clone(), W0.clone()
    ck = gpu.zeros(checkpoint_shape(37, shape), dtype=gpu.float64, device="cuda")
    forward_raw(cfg, D, W, dep, R_, t_, ck)
    gdep, gpose = gpu.zeros_like(dep), gpu.zeros((37, 12), dtype=gpu.float64, device="cuda")
    gD0, gW0 = gpu.empty_like(D0), gpu.empty_like(W0)
    backward_raw(cfg, gD_, gW_, D0, W0, ck, dep, R_, t_, gdep, gpose, gD0, gW0)
    got = [x.cpu().numpy() for x in (gdep, gpose, gD0, gW0)]
    for a, b in zip(got, want):
        b = np.asarray(b).reshape(a.shape)
        # sums of up to a few thousand terms in double
        assert np.abs(a - b).max() <= 1e-9 * max(np.abs(b).max(), 1e-30)
