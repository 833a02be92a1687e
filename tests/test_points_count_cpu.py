"""Point clouds that count more points than they hold (a slot extracted twice,
the old size set after a filter): the calls that would hand the count to a
kernel refuse it on the host.  No GPU: the Python class on CPU tensors with a
library that must not be called, the C++ class on stand-ins of the runtime."""
import os
import subprocess

import numpy as np
import pytest
import torch

from cuphoto import points as P
from cuphoto.points import PointCloud

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.join(HERE, "..")
K = [100.0, 0, 0, 0, 100.0, 0, 31.5, 23.5, 1.0]
POSE = np.array([1.0, 0, 0, 0, 0, 0, 0])


def cloud(held, counted, total=None):
    pc = PointCloud.__new__(PointCloud)
    pc.camera_matrix = list(K)
    pc.total_num_pts = held if total is None else total
    pc.num_pts = counted
    pc.has_rgb = False
    pc.device_pts = torch.zeros((held, 33), dtype=torch.uint8)
    return pc


class Library:
    """Stands in for the engine's library: records the calls."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return 0
        return call


@pytest.fixture
def library(monkeypatch):
    lib = Library()
    monkeypatch.setattr(P.L, "lib", lambda: lib)
    monkeypatch.setattr(P.L, "device_image", lambda t, *a, **kw: t)
    monkeypatch.setattr(P, "_stream_handle", lambda s: 0)
    return lib


@pytest.mark.parametrize("held,counted", [(6, 7), (6, 12), (0, 1)])
def test_counts_above_the_buffer_are_refused(library, capsys, held, counted):
    pc = cloud(held, counted)
    img = torch.zeros((2, 3))
    assert pc.transform(POSE) is False
    assert pc.project_to_depth(img, POSE) is False
    assert pc.project_to_color_depth(torch.zeros((2, 3, 3), dtype=torch.uint8), img, POSE) is False
    assert library.calls == []
    assert capsys.readouterr().err.count("%d points counted, %d held" % (counted, held)) == 3


def test_counts_up_to_the_buffer_reach_the_library(library):
    for counted in (1, 5, 6):
        assert cloud(6, counted).transform(POSE) is True
    assert [(n, a[1]) for n, a in library.calls] == [("gbt_points_transform", c) for c in (1, 5, 6)]


def test_extraction_is_given_the_buffer_s_capacity(library):
    """After a filter the buffer is smaller than the cloud was created with."""
    pc = cloud(4, 4, total=6)
    pc.extract_points(torch.zeros((2, 3)), None, POSE, 0)
    (name, args), = library.calls
    assert name == "gbt_points_extract" and args[12] == 4


def test_stored_count_is_that_of_the_points(tmp_path):
    pc = cloud(2, 4)
    assert pc.save_ply(str(tmp_path / "p.ply"))
    lines = (tmp_path / "p.ply").read_text().splitlines()
    assert lines[2] == "element vertex 2" and len(lines) == 10 + 2


CPP = r'''
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "cuphoto/cuda_point_cloud.cuh"

static int calls = 0;
static long long seen = -1;
extern "C" {
// the runtime on host memory, with guard bytes behind each allocation
cudaError_t cudaMallocManaged(void** p, size_t n, unsigned) { *p = std::malloc(n + 4096); std::memset(*p, 0xAB, n + 4096); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
const char* gbt_last_error(void) { return ""; }
gbt_status gbt_points_extract(const double*, const void*, int64_t, int32_t, float, const uint8_t*, int64_t, int32_t,
                              int32_t, const double*, int64_t, gbt_point*, int64_t capacity, void*) {
    ++calls;
    seen = capacity;
    return GBT_OK;
}
gbt_status gbt_points_transform(gbt_point*, int64_t n, const double*, void*) {
    ++calls;
    seen = n;
    return GBT_OK;
}
gbt_status gbt_points_project(const gbt_point*, int64_t n, const double*, const double*, float*, int64_t, uint8_t*,
                              int64_t, int32_t, int32_t, void*, void*) {
    ++calls;
    seen = n;
    return GBT_OK;
}
}

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main(int, char** argv) {
    using cuphoto::cudaPointCloud;
    std::array<double, 9> K = {100, 0, 0, 0, 100, 0, 1, 1, 1};
    std::array<double, 7> pose = {1, 0, 0, 0, 0, 0, 0};
    float img[6] = {};
    unsigned char rgb[18] = {};
    cv::cuda::PtrStepSzf depth(2, 3, img, 12);
    cv::cuda::PtrStepb none;
    cv::cuda::PtrStepSzb color(2, 3, rgb, 9);
    auto pc = cudaPointCloud::create(K, 6);
    CHECK(pc->extract_points(depth, none, pose, 0) && seen == 6);
    CHECK(pc->transform(pose) && pc->project_to_depth(depth, pose) && seen == 6);
    CHECK(pc->extract_points(depth, none, pose, 0));   // the same slot: counted twice
    CHECK(pc->get_num_points() == 12);
    const int before = calls;
    CHECK(!pc->transform(pose) && !pc->project_to_depth(depth, pose) && !pc->project_to_color_depth(color, depth, pose));
    auto other = cudaPointCloud::create(K, 2);
    CHECK(!other->add_point_cloud(pc) && !pc->add_point_cloud(other));
    CHECK(calls == before);
    CHECK(pc->save_ply(argv[1]));
    auto both = cudaPointCloud::merge(pc, other);
    for (int i = 0; i < 6; ++i) CHECK(std::memcmp(both->get_vertex(i), pc->get_vertex(i), 33) == 0);
    for (int i = 6; i < 12; ++i)
        for (int b = 0; b < 33; ++b) CHECK(reinterpret_cast<unsigned char*>(both->get_vertex(i))[b] == 0);
    pc->filter_depth();   // every z is 0, outside (min, max): all six are kept
    CHECK(pc->get_num_points() == 6 && pc->transform(pose) && seen == 6);
    for (int i = 0; i < 6; ++i) pc->get_vertex(i)->pos.z = i < 4 ? 1.f : 0.f;
    pc->filter_depth();   // two are kept, in a buffer of two
    CHECK(pc->get_num_points() == 2);
    pc->set_total_number_pts();
    CHECK(pc->get_num_points() == 6 && !pc->transform(pose));
    CHECK(pc->extract_points(depth, none, pose, 0) && seen == 2);   // (the engine refuses six in two)
    CHECK(!pc->add_vertex(make_float3(0, 0, 0), make_uchar3(0, 0, 0), 2));
    pc->clear();
    CHECK(reinterpret_cast<unsigned char*>(pc->get_vertex(2))[0] == 0xAB);
    std::printf("ok\n");
    return 0;
}
'''


def test_cpp_cloud_refuses_counts_above_its_buffer(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(CPP)
    pkg = os.path.join(ROOT, "cu-reconstruction_gb300", "cpp")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "t")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + os.path.join(pkg, "include"),
                           "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(cuda, "include"), str(src),
                           os.path.join(pkg, "src", "cuda_point_cloud.cpp"), "-o", exe])
    r = subprocess.run([exe, str(tmp_path / "p.ply")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
    lines = (tmp_path / "p.ply").read_text().splitlines()
    assert lines[2] == "element vertex 6" and len(lines) == 10 + 6
