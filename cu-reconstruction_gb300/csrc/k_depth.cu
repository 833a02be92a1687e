// Depth pyramids: per frame, the largest and the least positive depth of square
// tiles of pixels, which tell the integrate kernels the boxes of voxels that a
// frame cannot update and those that lie before all it sees (box_test in
// gbt_kernels.cuh).
#include <cstdint>
#include <cuda_runtime.h>

#include "gbt_internal.h"

namespace gbt {
namespace depth {

// The largest and the least positive depth so far.
struct Range {
    float far, least;
    __device__ __forceinline__ void add(float d) {
        far = fmaxf(far, d == d ? d : __int_as_float(0x7f800000));
        // (a subnormal is above 0 or not as the arithmetic flushes it: never "in front")
        least = fminf(least, d > 0.f ? (d < 1.17549435e-38f ? -3.0e38f : d) : 3.0e38f);
    }
    __device__ __forceinline__ void add(const float2& r) {
        far = fmaxf(far, r.x);
        least = fminf(least, r.y);
    }
};

// The 8 x 8 pixels at (x, y), x a multiple of 8: rows as 16-byte vectors where
// the whole tile is inside and they are aligned.  Samples in metres as the
// integrate kernels form them.
__device__ __forceinline__ Range tile_range(const FrameDesc& f, int x, int y) {
    Range m{0.f, 3.0e38f};
    const int rows = min(8, f.height - y), cols = min(8, f.width - x);
    const char* p = static_cast<const char*>(f.depth) + (int64_t)y * f.pitch;
    const bool vec = cols == 8 && rows == 8 && ((reinterpret_cast<uintptr_t>(f.depth) | (uintptr_t)f.pitch) & 15u) == 0;
    if (f.fmt == GBT_DEPTH_U16) {
        if (vec) {
            uint4 r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = __ldg(reinterpret_cast<const uint4*>(p + (int64_t)k * f.pitch + 2 * x));
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t w[4] = {r[k].x, r[k].y, r[k].z, r[k].w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    m.add(__fmul_rn((float)(w[q] & 0xffffu), f.scale));
                    m.add(__fmul_rn((float)(w[q] >> 16), f.scale));
                }
            }
        } else {
            for (int k = 0; k < rows; ++k)
                for (int q = 0; q < cols; ++q)
                    m.add(__fmul_rn((float)__ldg(reinterpret_cast<const unsigned short*>(p + (int64_t)k * f.pitch) + x + q),
                                    f.scale));
        }
    } else {
        if (vec) {
            float4 r[16];
#pragma unroll
            for (int k = 0; k < 16; ++k)
                r[k] = __ldg(reinterpret_cast<const float4*>(p + (int64_t)(k >> 1) * f.pitch + 4 * x) + (k & 1));
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                m.add(r[k].x);
                m.add(r[k].y);
                m.add(r[k].z);
                m.add(r[k].w);
            }
        } else {
            for (int k = 0; k < rows; ++k)
                for (int q = 0; q < cols; ++q)
                    m.add(__ldg(reinterpret_cast<const float*>(p + (int64_t)k * f.pitch) + x + q));
        }
    }
    return m;
}

// One CTA per 128 x 128 pixels of a frame, a thread per 8 x 8 of them, the
// coarser levels from shared memory.  The images are read once (0.6 MB for
// 640x480 uint16, 300 frames in about 40 us).
__device__ __forceinline__ void pyramid_block(const FrameDesc& f, float2* out) {
    __shared__ float2 s[16][17];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int bx = (int)blockIdx.x * 16, by = (int)blockIdx.y * 16;   // in tiles of 8 x 8
    int w = (f.width + 7) >> 3, h = (f.height + 7) >> 3;
    if (bx >= w || by >= h) return;   // the same for the whole CTA
    Range m{0.f, 3.0e38f};
    if (bx + tx < w && by + ty < h) {
        m = tile_range(f, 8 * (bx + tx), 8 * (by + ty));
        out[(by + ty) * w + bx + tx] = make_float2(m.far, m.least);
    }
    s[ty][tx] = make_float2(m.far, m.least);
#pragma unroll
    for (int l = 1; l < kPyrLevels; ++l) {
        out += w * h;
        w = (w + 1) >> 1;
        h = (h + 1) >> 1;
        const int n = 16 >> l;   // tiles of this level in the block, each way
        __syncthreads();
        if (tx < n && ty < n) {
            m = Range{0.f, 3.0e38f};
            m.add(s[2 * ty][2 * tx]);
            m.add(s[2 * ty][2 * tx + 1]);
            m.add(s[2 * ty + 1][2 * tx]);
            m.add(s[2 * ty + 1][2 * tx + 1]);
            const int x = (bx >> l) + tx, y = (by >> l) + ty;
            if (x < w && y < h) out[y * w + x] = make_float2(m.far, m.least);
        }
        __syncthreads();
        if (tx < n && ty < n) s[ty][tx] = make_float2(m.far, m.least);
    }
}

__global__ void __launch_bounds__(256) pyramid_table_kernel(const FrameDesc* frames, DepthPyr pyr) {
    pyramid_block(frames[blockIdx.z], const_cast<float2*>(pyr.of((int)blockIdx.z)));
}

__global__ void __launch_bounds__(256) pyramid_pass_kernel(const __grid_constant__ IntegrateArgs a) {
    asm volatile("griddepcontrol.launch_dependents;");   // the pass kernel's CTAs may take their places
    pyramid_block(a.frames[blockIdx.z], const_cast<float2*>(a.pyr.of((int)blockIdx.z)));
}

dim3 grid(int32_t width, int32_t height, int n) {
    return dim3((unsigned)(width + 127) / 128u, (unsigned)(height + 127) / 128u, (unsigned)n);
}

}  // namespace depth

cudaError_t launch_depth_pyramids(const FrameDesc* frames, int n, int32_t max_width, int32_t max_height,
                                  const DepthPyr& pyr, cudaStream_t s) {
    constexpr int kMaxZ = 65535;
    for (int f = 0; f < n; f += kMaxZ) {
        DepthPyr part = pyr;
        part.base += (size_t)f * pyr.stride;
        depth::pyramid_table_kernel<<<depth::grid(max_width, max_height, n - f < kMaxZ ? n - f : kMaxZ), 256, 0, s>>>(
            frames + f, part);
    }
    return cudaGetLastError();
}

cudaError_t launch_depth_pyramids(const IntegrateArgs& a, int32_t max_width, int32_t max_height, cudaStream_t s) {
    depth::pyramid_pass_kernel<<<depth::grid(max_width, max_height, a.nframes), 256, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace gbt
