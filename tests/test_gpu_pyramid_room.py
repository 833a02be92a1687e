"""Depth pyramids and the room for them.  The integrate calls of the C ABI take
the room that is there or go without, and allocate nothing; the reserve calls
(which the Python and C++ layers make) provide it, while streams are being
captured too.  With and without pyramids the volume is the same."""
import ctypes as C
import threading

import numpy as np
import pytest

from cuphoto import TSDFVolume, TSDFVolumeConfig, _lib as L
from cuphoto import synthetic as S
from cuphoto.batch import BatchIntegrator
from cuphoto.tsdf import make_frame

from helpers import dev_depth
from test_gpu_depth_cull import config, frames, volume_bits

pytestmark = pytest.mark.gpu

GRID = (144, 136, 140)   # 44 M voxel-frames with 16 frames


def counted(call):
    """(launches, frames) of depth pyramids in call()."""
    c = [L.debug_count(k) for k in (L.COUNT_PYRAMID_LAUNCHES, L.COUNT_PYRAMID_FRAMES)]
    call()
    return tuple(L.debug_count(k) - c[k] for k in (L.COUNT_PYRAMID_LAUNCHES, L.COUNT_PYRAMID_FRAMES))


def plain_integrate(vol, dd, poses, stream=None):
    """gbt_integrate without a reserve call."""
    arr = (L.Frame * len(dd))(*[make_frame(d, p) for d, p in zip(dd, poses)])
    L.check(L.lib().gbt_integrate(vol.handle, arr, len(dd), stream.cuda_stream if stream is not None else None))


def plain_batch(batch, vols, dds, poses, stream=None):
    """gbt_integrate_batch without a reserve call."""
    arr, items = [], (L.BatchItem * len(vols))()
    for k, (v, dd, ps) in enumerate(zip(vols, dds, poses)):
        items[k] = L.BatchItem(v.handle.value, len(arr), len(dd))
        arr += [make_frame(d, p) for d, p in zip(dd, ps)]
    L.check(L.lib().gbt_integrate_batch(batch._h, items, len(vols), (L.Frame * len(arr))(*arr), len(arr), 128, 0, 0,
                                        stream.cuda_stream if stream is not None else None))


@pytest.fixture(scope="module")
def half():
    return frames("frontal", "u16", 4)


@pytest.fixture(scope="module")
def hd():
    cam = S.Camera.hd()
    seq = S.make_sequence(16, scene_id=2, camera=cam, trajectory="frontal")
    return list(seq.depth_u16), seq.poses, cam


def want(gpu, tc, dd, poses):
    vol = TSDFVolume(tc)
    vol.integrate_frames(dd, poses, brick=4)   # without pyramids
    return volume_bits(gpu, vol)


def same(gpu, vol, bits):
    D, W = volume_bits(gpu, vol)
    return np.array_equal(D, bits[0]) and np.array_equal(W, bits[1])


@pytest.mark.parametrize("mode,arith", [("compat", "ieee"), ("fixed", "ieee"), ("compat", "reference")])
@pytest.mark.parametrize("camera", [(0, 0), (64, 48), (160, 120)])
def test_calls_without_room_go_without(gpu, half, camera, mode, arith):
    depths, poses, cam = half
    dd = [dev_depth(gpu, d) for d in depths]
    tc = config("frontal", GRID, cam, mode=mode, arith=arith, camera_width=camera[0], camera_height=camera[1])
    bits = want(gpu, tc, dd, poses)
    vol = TSDFVolume(tc)
    warm = TSDFVolume(tc)
    for call in (plain_integrate, lambda v, *a: v.integrate_frames(*a)):   # (kernels are loaded by their first launch)
        call(warm, dd, poses)
    gpu.cuda.synchronize()
    free = gpu.cuda.mem_get_info()[0]
    assert counted(lambda: plain_integrate(vol, dd, poses)) == (0, 0)
    gpu.cuda.synchronize()
    assert gpu.cuda.mem_get_info()[0] == free
    assert same(gpu, vol, bits)
    vol.reset()
    assert counted(lambda: vol.integrate_frames(dd, poses)) == (1, 16)   # the Python layer reserves
    assert same(gpu, vol, bits)
    vol.reset()
    assert counted(lambda: plain_integrate(vol, dd, poses)) == (1, 16)   # and what it reserved stays
    assert same(gpu, vol, bits)


def test_batched_calls_without_room_go_without(gpu, hd):
    depths, poses, cam = hd
    dd = [dev_depth(gpu, d) for d in depths]
    tc = config("frontal", GRID, cam, mode="fixed")
    bits = want(gpu, tc, dd, poses)
    vol = TSDFVolume(tc)
    plain_batch(BatchIntegrator(1, 16), [vol], [dd], [poses])   # (kernels are loaded by their first launch)
    vol.reset()
    batch = BatchIntegrator(1, 16)
    gpu.cuda.synchronize()
    free = gpu.cuda.mem_get_info()[0]
    assert counted(lambda: plain_batch(batch, [vol], [dd], [poses])) == (0, 0)
    gpu.cuda.synchronize()
    assert gpu.cuda.mem_get_info()[0] == free
    assert same(gpu, vol, bits)
    vol.reset()
    assert counted(lambda: batch.integrate([vol], [dd], [poses])) == (1, 16)
    assert same(gpu, vol, bits)


@pytest.mark.parametrize("reserve", [False, True])
@pytest.mark.parametrize("batched", [False, True])
def test_graphs_without_pyramids_and_with_an_outgrown_buffer(gpu, half, hd, batched, reserve):
    """Captured on objects that have too little room: without pyramids, or after a
    reserve call under capture.  Replayed as captured, and once more after a
    larger call has moved the buffer."""
    depths, poses, cam = hd if batched else half
    dd = [dev_depth(gpu, d) for d in depths]
    tc = config("frontal", GRID, cam, camera_width=64, camera_height=48)
    bits = want(gpu, tc, dd, poses)
    vol, other = TSDFVolume(tc), TSDFVolume(tc)
    batch, larger = BatchIntegrator(1, 16), BatchIntegrator(1, 16)
    s, g = gpu.cuda.Stream(), gpu.cuda.CUDAGraph()

    def record():
        with gpu.cuda.graph(g, stream=s):
            if batched and reserve:
                batch.integrate([vol], [dd], [poses], stream=s)
            elif batched:
                plain_batch(batch, [vol], [dd], [poses], s)
            elif reserve:
                vol.integrate_frames(dd, poses, stream=s)
            else:
                plain_integrate(vol, dd, poses, s)

    assert counted(record) == ((1, 16) if reserve else (0, 0))
    g.replay()
    assert same(gpu, vol, bits)
    if batched:   # (a graph reads the staging area of its batch's last call: another batch grows)
        larger.integrate([other], [dd], [poses])
    else:
        vol.integrate_frames(dd + dd, list(poses) + list(poses))
    vol.reset()
    gpu.cuda.synchronize()
    g.replay()
    assert same(gpu, vol, bits)


def test_without_memory_for_pyramids(gpu, half):
    depths, poses, cam = half
    dd = [dev_depth(gpu, d) for d in depths]
    tc = config("frontal", GRID, cam, camera_width=0, camera_height=0)
    bits = want(gpu, tc, dd, poses)
    vol = TSDFVolume(tc)
    try:
        L.lib().gbt_debug_inject(L.INJECT_ALLOC, 0, 1)
        assert counted(lambda: vol.integrate_frames(dd, poses)) == (0, 0)
    finally:
        L.lib().gbt_debug_inject(L.INJECT_NONE, 0, 0)
    assert same(gpu, vol, bits)
    arr = (L.Frame * 16)(*[make_frame(d, p) for d, p in zip(dd, poses)])
    assert L.lib().gbt_volume_reserve(vol.handle, arr, 16) == L.GBT_OK
    vol.reset()
    assert counted(lambda: vol.integrate_frames(dd, poses)) == (1, 16)
    assert same(gpu, vol, bits)


def test_growth_does_not_end_another_thread_s_capture(gpu, half):
    """A capture in global mode forbids other threads' allocations, unless they
    are marked as harmless to it."""
    depths, poses, cam = half
    dd = [dev_depth(gpu, d) for d in depths]
    tc = config("frontal", GRID, cam, camera_width=64, camera_height=48)
    bits = want(gpu, tc, dd, poses)
    a, b = TSDFVolume(tc), TSDFVolume(tc)
    s, t, g = gpu.cuda.Stream(), gpu.cuda.Stream(), gpu.cuda.CUDAGraph()
    failed = []

    def work():
        try:
            b.integrate_frames(dd, poses, stream=t)
        except Exception as e:
            failed.append(e)

    gpu.cuda.synchronize()
    with gpu.cuda.graph(g, stream=s, capture_error_mode="global"):
        a.integrate_frames(dd, poses, stream=s)
        th = threading.Thread(target=work)
        th.start()
        th.join()
    assert not failed
    g.replay()
    assert same(gpu, a, bits) and same(gpu, b, bits)


def test_reserve_calls_check_their_arguments(gpu, half):
    depths, poses, cam = half
    vol = TSDFVolume(config("frontal", (16, 16, 16), cam))
    f = make_frame(dev_depth(gpu, depths[0]), poses[0])
    lib = L.lib()
    assert lib.gbt_volume_reserve(None, C.byref(f), 1) == L.GBT_ERR_INVALID_ARG
    for n in (0, 33):
        assert lib.gbt_volume_reserve(vol.handle, (L.Frame * 33)(f), n) == L.GBT_ERR_INVALID_ARG
    bad = L.Frame()
    assert lib.gbt_volume_reserve(vol.handle, C.byref(bad), 1) == L.GBT_ERR_INVALID_ARG
    batch = BatchIntegrator(1, 2)
    ok = (L.Frame * 2)(f, f)
    for items in ([(None, 0, 1)], [(vol.handle.value, 0, 3)], [(vol.handle.value, -1, 1)], [(vol.handle.value, 0, 1)] * 2):
        it = (L.BatchItem * len(items))(*[L.BatchItem(*i) for i in items])
        assert lib.gbt_batch_reserve(batch._h, it, len(items), ok, 2) == L.GBT_ERR_INVALID_ARG
    one = (L.BatchItem * 1)(L.BatchItem(vol.handle.value, 0, 2))
    assert lib.gbt_batch_reserve(batch._h, one, 1, ok, 3) == L.GBT_ERR_INVALID_ARG
    assert lib.gbt_batch_reserve(batch._h, one, 1, ok, 2) == L.GBT_OK
    n = C.c_int64()
    assert lib.gbt_debug_count(7, C.byref(n)) == L.GBT_ERR_INVALID_ARG
    assert lib.gbt_debug_count(0, None) == L.GBT_ERR_INVALID_ARG


def test_creation_without_memory_for_pyramids(gpu, half, hd):
    """The room is optional: its allocation, the last of a volume's or batch's,
    may fail."""
    depths, poses, cam = half
    dd = [dev_depth(gpu, d) for d in depths]
    tc = config("frontal", GRID, cam)
    bits = want(gpu, tc, dd, poses)
    made = []
    try:
        for create in (lambda: TSDFVolume(tc), lambda: BatchIntegrator(1, 16)):
            L.lib().gbt_debug_inject(L.INJECT_ALLOC, 2, 1)
            made.append(create())
    finally:
        L.lib().gbt_debug_inject(L.INJECT_NONE, 0, 0)
    vol, batch = made
    assert counted(lambda: plain_integrate(vol, dd, poses)) == (0, 0)
    assert same(gpu, vol, bits)
    vol.reset()
    assert counted(lambda: plain_batch(batch, [vol], [dd], [poses])) == (0, 0)
    assert same(gpu, vol, bits)
    vol.reset()
    assert counted(lambda: batch.integrate([vol], [dd], [poses])) == (1, 16)
    assert same(gpu, vol, bits)


@pytest.mark.parametrize("grid,camera,frames_with_room", [
    ((160, 160, 160), (640, 480), 32),
    ((160, 160, 160), (1280, 720), 32),
    ((400, 400, 400), (2560, 1920), 32),
    ((240, 232, 236), (4096, 4096), 0),   # pyramids pay in no pass of such frames into these
    ((96, 80, 72), (640, 480), 0),
    ((64, 64, 64), (4096, 4096), 0)])
def test_room_at_creation_is_that_of_the_grid(gpu, grid, camera, frames_with_room):
    """How many frames of the configured camera one pass can have pyramids of,
    without a reserve call; larger passes go without."""
    w, h = camera
    vol = TSDFVolume(config("circle", grid, S.Camera.half(), camera_width=w, camera_height=h))
    img = gpu.zeros((h, w), dtype=gpu.int16, device="cuda")
    pose = S.circle_poses(8)[0]
    most = 0
    for n in range(1, 33):
        c = counted(lambda: plain_integrate(vol, [img] * n, [pose] * n))
        if c == (1, n):
            most = n
    assert most == frames_with_room


def test_frames_that_no_item_takes_get_no_pyramid(gpu, half):
    """A long table of which the items take a few ranges."""
    depths, poses, cam = half
    dd = [dev_depth(gpu, d) for d in depths]
    n = len(dd)
    tc = config("frontal", GRID, cam, mode="fixed")
    vols = [TSDFVolume(tc) for _ in range(3)]
    ranges = [(7, 9), (20, 5), (24, 6)]         # frames 7-15, 20-24 and 24-29 of 40
    table = [make_frame(dd[k % n], poses[k % n]) for k in range(40)]
    for k in range(40):
        if not any(a <= k < a + c for a, c in ranges):
            table[k].width = table[k].height = 1   # small images: none of them is read
            table[k].pitch_bytes = 2
    items = (L.BatchItem * 3)(*[L.BatchItem(v.handle.value, a, c) for v, (a, c) in zip(vols, ranges)])
    batch = BatchIntegrator(3, 40)
    st = counted(lambda: L.check(L.lib().gbt_integrate_batch(batch._h, items, 3, (L.Frame * 40)(*table), 40, 128, 0, 0,
                                                             None)))
    assert st == (1, 9 + 5 + 6 - 1)
    for v, (a, c) in zip(vols, ranges):
        k = [i % n for i in range(a, a + c)]
        assert same(gpu, v, want(gpu, tc, [dd[i] for i in k], [poses[i] for i in k]))


@pytest.mark.parametrize("height,with_pyramid", [(65535 * 128, 1), (65535 * 128 + 1, 0)])
def test_images_taller_than_a_grid_of_blocks(gpu, height, with_pyramid):
    """An image of one column and more rows than one launch's blocks cover is
    integrated without a pyramid, by single passes and by the batch."""
    n, w = 312, 1
    tc = TSDFVolumeConfig(voxel_grid_size=(n, n, n), physical_size=(1.0, 1.0, 1.0), global_offset=(-0.5, -0.5, 0.5),
                          focal_x=0.75, focal_y=200.0, cx=0.0, cy=150.0, camera_width=w, camera_height=300, mode="fixed")
    img = gpu.full((height, w), 1000, dtype=gpu.int16, device="cuda")
    img[100:130] = 0
    pose = np.array([1.0, 0, 0, 0, 0, 0, 0])
    bits = want(gpu, tc, [img], [pose])
    assert (bits[1] > 0).mean() > 0.1
    vol = TSDFVolume(tc)
    assert counted(lambda: vol.integrate(img, img, pose)) == (with_pyramid, with_pyramid)
    assert same(gpu, vol, bits)
    vol.reset()
    batch = BatchIntegrator(1, 1)
    assert counted(lambda: batch.integrate([vol], [[img]], [[pose]])) == (with_pyramid, with_pyramid)
    assert same(gpu, vol, bits)


@pytest.mark.parametrize("first,count", [(2 ** 31 - 1, 1), (1, 2 ** 31 - 1), (2, 1), (0, 3), (-1, 1), (0, -1)])
def test_item_ranges_outside_the_table_are_refused(gpu, half, first, count):
    """Ranges whose end does not fit an int32 among them."""
    depths, poses, cam = half
    vol = TSDFVolume(config("frontal", (16, 16, 16), cam))
    batch = BatchIntegrator(1, 2)
    table = (L.Frame * 2)(*[make_frame(dev_depth(gpu, depths[0]), poses[0])] * 2)
    items = (L.BatchItem * 1)(L.BatchItem(vol.handle.value, first, count))
    for st in (L.lib().gbt_batch_reserve(batch._h, items, 1, table, 2),
               L.lib().gbt_integrate_batch(batch._h, items, 1, table, 2, 128, 0, 0, None)):
        assert st == L.GBT_ERR_INVALID_ARG and b"outside the frame table" in L.lib().gbt_last_error()
