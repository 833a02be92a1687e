"""Integrate with depth pyramids (calls of 8 M voxel-frames and more) against
the CPU oracle and against the passes that go without them (bricks 4-7), bit
for bit, on frames made to trip the culling: holes, frames without depth, lone
far pixels, unusable values (NaN, infinite, negative, beyond the usable range),
images of several sizes and alignments, cameras inside the volume."""
import numpy as np
import pytest

from cuphoto import TSDFVolume, TSDFVolumeConfig
from cuphoto import synthetic as S
from cuphoto.batch import BatchIntegrator

from helpers import dev_depth, oracle_run

pytestmark = pytest.mark.gpu

GRIDS = [(96, 80, 72), (93, 81, 74)]


def frames(path, fmt, seed, n=16):
    cam = S.Camera.half()
    seq = S.make_sequence(n, scene_id=seed, camera=cam, trajectory=path)
    rng = np.random.default_rng(seed)
    out = []
    for k in range(n):
        raw = seq.depth_u16[k].copy()
        for _ in range(6):   # holes with straight edges, some over whole tiles
            y, x = rng.integers(0, cam.height), rng.integers(0, cam.width)
            raw[y:y + rng.integers(1, 70), x:x + rng.integers(1, 90)] = 0
        if k == 1:
            raw[:] = 0
        if k == 2:
            raw[:] = 500
            raw[rng.random(raw.shape) < 0.002] = 4000       # lone far pixels
        if k == 3:
            raw[rng.random(raw.shape) < 0.01] = 65535        # beyond 24 m
        d = raw if fmt == "u16" else raw.astype(np.float32) * np.float32(0.001)
        if fmt == "f32" and k == 4:
            d[rng.random(d.shape) < 0.3] = np.nan
            d[rng.random(d.shape) < 0.1] = np.inf
            d[rng.random(d.shape) < 0.1] = -1.0
        if fmt == "f32" and k == 8:
            d[rng.random(d.shape) < 0.01] = 1e-40            # subnormal: 0 where the arithmetic flushes
            d[rng.random(d.shape) < 0.01] = -0.0
        if k == 5:
            d = d[:203, :317]                                # rows that start anywhere
        if k == 6:
            d = d[:8, :8]
        if k == 7:
            d = d[:1, :]
        out.append(np.ascontiguousarray(d))
    return out, seq.poses, cam


def config(path, grid, cam, **kw):
    g = S.frontal_grid(*grid) if path == "frontal" else dict(voxel_grid_size=grid, physical_size=(2.56,) * 3,
                                                             global_offset=(-1.28,) * 3)
    return TSDFVolumeConfig(**g, focal_x=cam.fx, focal_y=cam.fy, cx=cam.cx, cy=cam.cy, **kw)


def volume_bits(gpu, vol):
    gpu.cuda.synchronize()
    return (vol.voxel_distances_data().cpu().numpy().view(np.uint32).copy(),
            vol.voxel_weights_data().cpu().numpy().copy())


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("fmt", ["u16", "f32"])
@pytest.mark.parametrize("path", ["frontal", "circle"])
@pytest.mark.parametrize("mode,arith", [("compat", "ieee"), ("fixed", "ieee"), ("compat", "reference")])
def test_passes_and_batches_with_pyramids(gpu, oracle, grid, fmt, path, mode, arith):
    depths, poses, cam = frames(path, fmt, 2)
    tc = config(path, grid, cam, mode=mode, arith=arith)
    dd = [dev_depth(gpu, d) for d in depths]
    assert np.prod(grid) * len(dd) >= 8 << 20
    plain = TSDFVolume(tc)
    plain.integrate_frames(dd, poses, brick=4)     # depth staged in shared memory: no pyramids
    D0, W0 = volume_bits(gpu, plain)
    assert (W0 > 0).any() and (W0 == 0).any()
    for brick in range(4):
        vol = TSDFVolume(tc)
        vol.integrate_frames(dd, poses, brick=brick)
        D, W = volume_bits(gpu, vol)
        assert np.array_equal(W, W0) and np.array_equal(D, D0), brick
        vol.reset()
        BatchIntegrator(1, 64).integrate([vol], [dd], [poses], brick=brick)
        D, W = volume_bits(gpu, vol)
        assert np.array_equal(W, W0) and np.array_equal(D, D0), brick
    vol = TSDFVolume(tc)
    vol.integrate_frames(dd + dd, list(poses) + list(poses))          # one frame per lane
    plain.integrate_frames(dd, poses, brick=4)
    D1, W1 = volume_bits(gpu, plain)
    D, W = volume_bits(gpu, vol)
    assert np.array_equal(W, W1) and np.array_equal(D, D1)
    if arith == "ieee":
        Do, Wo = oracle_run(oracle, tc, depths, poses)
        assert np.array_equal(W0, Wo) and np.array_equal(D0, Do.view(np.uint32))


def test_negative_scale_and_short_range(gpu, oracle):
    """uint16 with a negative scale has no usable sample; a fixed-mode volume
    with a short range beside one with a long one in the same batch."""
    depths, poses, cam = frames("circle", "u16", 3)
    dd = [dev_depth(gpu, d) for d in depths]
    near = config("circle", (96, 80, 72), cam, mode="fixed", max_depth=1.4)
    far = config("circle", (96, 80, 72), cam, mode="fixed", max_depth=9.0)
    a, b = TSDFVolume(near), TSDFVolume(far)
    BatchIntegrator(2, 64).integrate([a, b], [dd, dd], [poses, poses])
    for vol, tc in ((a, near), (b, far)):
        D, W = volume_bits(gpu, vol)
        Do, Wo = oracle_run(oracle, tc, depths, poses)
        assert np.array_equal(W, Wo) and np.array_equal(D, Do.view(np.uint32))
    D0, W0 = volume_bits(gpu, a)
    a.integrate_frames(dd, poses, depth_scale=-0.001)
    D, W = volume_bits(gpu, a)
    assert np.array_equal(W, W0) and np.array_equal(D, D0)


def test_graph_capture_before_and_after_pyramids_have_room(gpu):
    """Captured with and without a buffer for pyramids (one cannot be allocated
    while capturing), and replayed after a larger call moved the buffer."""
    depths, poses, cam = frames("frontal", "u16", 4)
    tc = config("frontal", (96, 80, 72), cam)
    dd = [dev_depth(gpu, d) for d in depths]
    ref = TSDFVolume(tc)
    ref.integrate_frames(dd, poses, brick=4)
    want = volume_bits(gpu, ref)
    for warm in (False, True):
        vol = TSDFVolume(tc)
        if warm:
            vol.integrate_frames(dd, poses)
        s = gpu.cuda.Stream()
        g = gpu.cuda.CUDAGraph()
        with gpu.cuda.graph(g, stream=s):
            vol.integrate_frames(dd, poses, stream=s)
        if warm:   # more frames than the buffer had room for
            vol.integrate_frames(dd + dd, list(poses) + list(poses))
        vol.reset()
        gpu.cuda.synchronize()
        g.replay()
        D, W = volume_bits(gpu, vol)
        assert np.array_equal(D, want[0]) and np.array_equal(W, want[1])


@pytest.mark.parametrize("nz", [1, 3, 4, 5, 71])
@pytest.mark.parametrize("nx", [1, 31, 36, 65])
@pytest.mark.parametrize("mode,arith", [("compat", "ieee"), ("fixed", "ieee"), ("compat", "reference")])
def test_voxel_runs_along_x_and_z(gpu, oracle, nx, nz, mode, arith):
    """Passes whose threads hold voxels along x or along z, and the batched
    kernel (along z) of one and of two volumes, at extents around their runs."""
    depths, poses, cam = frames("circle", "u16", 5, n=9)
    depths = [d for d in depths if d.shape == depths[0].shape]
    poses = poses[:len(depths)]
    tc = config("circle", (nx, 18, nz), cam, mode=mode, arith=arith)
    dd = [dev_depth(gpu, d) for d in depths]
    want = TSDFVolume(tc)
    for d, p in zip(dd, poses):
        want.integrate_frames([d], [p], brick=5)
    D0, W0 = volume_bits(gpu, want)
    for k in (1, 2, 5, 6):
        vol = TSDFVolume(tc)
        vol.integrate_sequence(dd, poses, frames_per_pass=k, brick=k % 4)
        D, W = volume_bits(gpu, vol)
        assert np.array_equal(W, W0) and np.array_equal(D, D0), k
    vols = [TSDFVolume(tc), TSDFVolume(config("circle", (40, 18, 8), cam, mode=mode, arith=arith))]
    for n in (1, 2):
        for vol in vols:
            vol.reset()
        for brick in range(4):
            vols[0].reset()
            BatchIntegrator(2, 64).integrate(vols[:n], [dd] * n, [poses] * n, brick=brick)
            D, W = volume_bits(gpu, vols[0])
            assert np.array_equal(W, W0) and np.array_equal(D, D0), (n, brick)
    if arith == "ieee":
        Do, Wo = oracle_run(oracle, tc, depths, poses)
        assert np.array_equal(W0, Wo) and np.array_equal(D0, Do.view(np.uint32))
