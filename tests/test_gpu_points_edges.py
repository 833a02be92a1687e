"""The point-cloud kernels where their loads and stores change form: clouds
that start on any byte, counts around the ends of a warp and a CTA."""
import ctypes as C

import numpy as np
import pytest

from cuphoto import synthetic as S

pytestmark = pytest.mark.gpu


def cloud(oracle, n, seed):
    rng = np.random.default_rng(seed)
    pts = np.zeros((n, 33), np.uint8)
    v = pts.reshape(-1).view(oracle.POINT_DTYPE)
    v["pos"] = rng.normal(scale=0.6, size=(n, 3)).astype(np.float32)
    v["normal"] = rng.normal(size=(n, 4)).astype(np.float32)
    v["color"] = rng.integers(0, 256, (n, 3))
    v["class_id"] = rng.integers(0, 65536, n)
    return pts


def at_byte(torch, pts, offset):
    """The records on the GPU from byte `offset` of an allocation, 0xAB around them."""
    n = pts.nbytes
    buf = torch.full((n + 64,), 0xAB, dtype=torch.uint8, device="cuda")
    buf[offset:offset + n] = torch.from_numpy(pts.reshape(-1)).cuda()
    return buf, buf[offset:offset + n]


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 16])
@pytest.mark.parametrize("n", [1, 2, 5, 31, 32, 33, 255, 256, 257, 5003])
def test_project_from_any_byte(gpu, engine_lib, oracle, offset, n):
    pts = cloud(oracle, n, 100 * n + offset)
    buf, dev = at_byte(gpu, pts, offset)
    w, h = 83, 61
    K = np.array([50.0, 0, 41.0, 0, 50.0, 30.0, 0, 0, 1.0])
    pose = S.circle_poses(8)[3]
    depth = gpu.full((h, w), 7.0, dtype=gpu.float32, device="cuda")
    rgb = gpu.full((h, w, 3), 9, dtype=gpu.uint8, device="cuda")
    scratch = gpu.empty(w * h, dtype=gpu.int64, device="cuda")
    engine_lib.check(engine_lib.lib().gbt_points_project(
        C.c_void_p(dev.data_ptr()), n, C.byref((C.c_double * 9)(*K)), C.byref((C.c_double * 7)(*pose)),
        C.c_void_p(depth.data_ptr()), 4 * w, C.c_void_p(rgb.data_ptr()), 3 * w, w, h,
        C.c_void_p(scratch.data_ptr()), None))
    gpu.cuda.synchronize()
    ed, ec = oracle.points_project(pts, K, pose, w, h)
    assert np.array_equal(depth.cpu().numpy().view(np.uint32), ed.view(np.uint32))
    assert np.array_equal(rgb.cpu().numpy(), ec)
    assert (ed > 0).any() or n < 31


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 8, 16])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 16, 255, 256, 257, 1000])
def test_transform_from_any_byte(gpu, engine_lib, oracle, offset, n):
    """Every byte of the records, and none outside them."""
    pts = cloud(oracle, n, 7 * n + offset)
    buf, dev = at_byte(gpu, pts, offset)
    pose = np.concatenate([[0.5, -0.5, 0.5, 0.5], [0.3, -1.2, 2.0]])
    engine_lib.check(engine_lib.lib().gbt_points_transform(C.c_void_p(dev.data_ptr()), n,
                                                           C.byref((C.c_double * 7)(*pose)), None))
    gpu.cuda.synchronize()
    oracle.points_transform(pts, pose)
    exp = np.full(pts.nbytes + 64, 0xAB, np.uint8)
    exp[offset:offset + pts.nbytes] = pts.reshape(-1)
    assert np.array_equal(buf.cpu().numpy(), exp)


@pytest.mark.parametrize("offset", [0, 1, 4, 16])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 1), (33, 3), (64, 8), (257, 5)])
@pytest.mark.parametrize("fx,cx", [(525.0, 319.5), (-313.7, 30.0 + 1e-9), (1.0 / 3, 16.0 - 2.0 ** -30), (2.0 ** 21, 7.25),
                                   (2.0 ** -21, 0.0)])
def test_extract_any_start_and_camera(gpu, engine_lib, oracle, offset, w, h, fx, cx):
    """Spans that do and do not start on 16 bytes, runs with and without depth,
    centres next to a pixel, focal lengths on both sides of the limits of the
    form without FP64, depths far outside a sensor's range."""
    rng = np.random.default_rng(w * 1000 + h)
    d = (rng.integers(1, 9000, (h, w)) * np.float32(0.001)).astype(np.float32)
    odd = np.array([1e-12, 3e-9, 2.0 ** -30, 2e9, 1e30, np.inf, 1.5, 0.75, 1e-38, np.nan], np.float32)
    d = np.where(rng.random((h, w)) < 0.2, odd[rng.integers(0, len(odd), (h, w))], d)
    d[rng.random((h, w)) < (0.5 if h == 3 else 0.1)] = 0
    rgb = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    pose = np.concatenate([[0.5, -0.5, 0.5, 0.5], [0.3, -1.2, 2.0]])
    K = np.array([fx, 0, 0, 0, 1.5 * fx, 0, cx, 0.5 * cx, 1.0])
    start, n = 3, w * h + 5
    exp = cloud(oracle, n, 11)
    buf, dev = at_byte(gpu, exp, offset)
    d_t, rgb_t = gpu.from_numpy(d).cuda(), gpu.from_numpy(rgb).cuda()
    engine_lib.check(engine_lib.lib().gbt_points_extract(
        C.byref((C.c_double * 9)(*K)), C.c_void_p(d_t.data_ptr()), 4 * w, engine_lib.DEPTH_F32_M, 1.0,
        C.c_void_p(rgb_t.data_ptr()), 3 * w, w, h, C.byref((C.c_double * 7)(*pose)), start,
        C.c_void_p(dev.data_ptr()), n, None))
    gpu.cuda.synchronize()
    got = buf.cpu().numpy()
    assert (got[:offset] == 0xAB).all() and (got[offset + exp.nbytes:] == 0xAB).all()
    oracle.points_extract(K, d, rgb, pose, exp, start=start)
    a, b = (r.reshape(-1).copy().view(oracle.POINT_DTYPE) for r in (got[offset:offset + exp.nbytes], exp))
    nan = np.isnan(a["pos"]) & np.isnan(b["pos"])   # (the payload of a NaN is the processor's)
    a["pos"][nan] = b["pos"][nan] = 0
    assert a.tobytes() == b.tobytes()


def test_extract_runs_from_a_vector_boundary(gpu, engine_lib, oracle):
    """The 16-byte form over every mix of pixels with and without depth in a span."""
    w, h = 32, 512
    rng = np.random.default_rng(5)
    d = (rng.integers(1, 9000, (h, w)) * np.float32(0.001)).astype(np.float32)
    for r in range(h):
        if r % 4 == 1:
            d[r, rng.random(w) < rng.random()] = 0
        elif r % 4 == 2:
            d[r, : r % 33] = 0
        elif r % 4 == 3:
            d[r, r % 33:] = 0
    pose = np.concatenate([[0.5, -0.5, 0.5, 0.5], [0.3, -1.2, 2.0]])
    K = np.array([525.0, 0, 0, 0, 525.0, 0, 319.5, 239.5, 1.0])
    exp = cloud(oracle, w * h, 12)
    buf, dev = at_byte(gpu, exp, 0)
    d_t = gpu.from_numpy(d).cuda()
    engine_lib.check(engine_lib.lib().gbt_points_extract(
        C.byref((C.c_double * 9)(*K)), C.c_void_p(d_t.data_ptr()), 4 * w, engine_lib.DEPTH_F32_M, 1.0, None, 0, w, h,
        C.byref((C.c_double * 7)(*pose)), 0, C.c_void_p(dev.data_ptr()), w * h, None))
    gpu.cuda.synchronize()
    oracle.points_extract(K, d, None, pose, exp)
    assert np.array_equal(buf.cpu().numpy()[:exp.nbytes], exp.reshape(-1))
