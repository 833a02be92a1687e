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
