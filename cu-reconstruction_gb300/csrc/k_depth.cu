// Depth pyramids: per frame, the largest usable depth of square tiles of pixels,
// which lets the integrate kernels cull the boxes of voxels that a frame cannot
// update (box_culled in gbt_kernels.cuh).
#include <cstdint>
#include <cuda_runtime.h>

#include "gbt_internal.h"

namespace gbt {
namespace depth {

// A depth sample in metres as the integrate kernels form it, 0 where they would
// not use it (not above 0, above the cap, or NaN).
__device__ __forceinline__ float usable(float d, float cap) { return d > 0.f && d <= cap ? d : 0.f; }

// The largest usable depth of the 8 x 8 pixels at (x, y), x a multiple of 8:
// rows as 16-byte vectors where the whole tile is inside and they are aligned.
__device__ __forceinline__ float tile_max(const FrameDesc& f, int x, int y, float cap) {
    float m = 0.f;
    const int rows = min(8, f.height - y), cols = min(8, f.width - x);
    const char* p = static_cast<const char*>(f.depth) + (int64_t)y * f.pitch;
    const bool vec = cols == 8 && ((reinterpret_cast<uintptr_t>(f.depth) | (uintptr_t)f.pitch) & 15u) == 0;
    if (f.fmt == GBT_DEPTH_U16) {
        if (vec && rows == 8) {
            uint4 r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = __ldg(reinterpret_cast<const uint4*>(p + (int64_t)k * f.pitch + 2 * x));
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t w[4] = {r[k].x, r[k].y, r[k].z, r[k].w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    m = fmaxf(m, usable(__fmul_rn((float)(w[q] & 0xffffu), f.scale), cap));
                    m = fmaxf(m, usable(__fmul_rn((float)(w[q] >> 16), f.scale), cap));
                }
            }
        } else {
            for (int k = 0; k < rows; ++k)
                for (int q = 0; q < cols; ++q) {
                    const float raw = (float)__ldg(reinterpret_cast<const unsigned short*>(p + (int64_t)k * f.pitch) + x + q);
                    m = fmaxf(m, usable(__fmul_rn(raw, f.scale), cap));
                }
        }
    } else {
        if (vec && rows == 8) {
            float4 r[16];
#pragma unroll
            for (int k = 0; k < 16; ++k)
                r[k] = __ldg(reinterpret_cast<const float4*>(p + (int64_t)(k >> 1) * f.pitch + 4 * x) + (k & 1));
#pragma unroll
            for (int k = 0; k < 16; ++k)
                m = fmaxf(m, fmaxf(fmaxf(usable(r[k].x, cap), usable(r[k].y, cap)),
                                   fmaxf(usable(r[k].z, cap), usable(r[k].w, cap))));
        } else {
            for (int k = 0; k < rows; ++k)
                for (int q = 0; q < cols; ++q)
                    m = fmaxf(m, usable(__ldg(reinterpret_cast<const float*>(p + (int64_t)k * f.pitch) + x + q), cap));
        }
    }
    return m;
}

// One CTA per 128 x 128 pixels of a frame, a thread per 8 x 8 of them, the
// coarser levels from shared memory.  The images are read once (0.6 MB for
// 640x480 uint16, 300 frames in about 40 us).
__device__ __forceinline__ void pyramid_block(const FrameDesc& f, float cap, float* out) {
    __shared__ float s[16][17];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int bx = (int)blockIdx.x * 16, by = (int)blockIdx.y * 16;   // in tiles of 8 x 8
    int w = (f.width + 7) >> 3, h = (f.height + 7) >> 3;
    if (bx >= w || by >= h) return;   // the same for the whole CTA
    float m = 0.f;
    if (bx + tx < w && by + ty < h) {
        m = tile_max(f, 8 * (bx + tx), 8 * (by + ty), cap);
        out[(by + ty) * w + bx + tx] = m;
    }
    s[ty][tx] = m;
#pragma unroll
    for (int l = 1; l < kPyrLevels; ++l) {
        out += w * h;
        w = (w + 1) >> 1;
        h = (h + 1) >> 1;
        const int n = 16 >> l;   // tiles of this level in the block, each way
        __syncthreads();
        if (tx < n && ty < n) {
            m = fmaxf(fmaxf(s[2 * ty][2 * tx], s[2 * ty][2 * tx + 1]), fmaxf(s[2 * ty + 1][2 * tx], s[2 * ty + 1][2 * tx + 1]));
            const int x = (bx >> l) + tx, y = (by >> l) + ty;
            if (x < w && y < h) out[y * w + x] = m;
        }
        __syncthreads();
        if (tx < n && ty < n) s[ty][tx] = m;
    }
}

__global__ void __launch_bounds__(256) pyramid_table_kernel(const FrameDesc* frames, float cap, DepthPyr pyr) {
    pyramid_block(frames[blockIdx.z], cap, const_cast<float*>(pyr.of((int)blockIdx.z)));
}

__global__ void __launch_bounds__(256) pyramid_pass_kernel(const __grid_constant__ IntegrateArgs a, float cap) {
    pyramid_block(a.frames[blockIdx.z], cap, const_cast<float*>(a.pyr.of((int)blockIdx.z)));
}

dim3 grid(int32_t width, int32_t height, int n) {
    return dim3((unsigned)(width + 127) / 128u, (unsigned)(height + 127) / 128u, (unsigned)n);
}

}  // namespace depth

cudaError_t launch_depth_pyramids(const FrameDesc* frames, int n, int32_t max_width, int32_t max_height, float cap,
                                  const DepthPyr& pyr, cudaStream_t s) {
    constexpr int kMaxZ = 65535;
    for (int f = 0; f < n; f += kMaxZ) {
        DepthPyr part = pyr;
        part.base += (size_t)f * pyr.stride;
        depth::pyramid_table_kernel<<<depth::grid(max_width, max_height, n - f < kMaxZ ? n - f : kMaxZ), 256, 0, s>>>(
            frames + f, cap, part);
    }
    return cudaGetLastError();
}

cudaError_t launch_depth_pyramids(const IntegrateArgs& a, int32_t max_width, int32_t max_height, float cap,
                                  cudaStream_t s) {
    depth::pyramid_pass_kernel<<<depth::grid(max_width, max_height, a.nframes), 256, 0, s>>>(a, cap);
    return cudaGetLastError();
}

}  // namespace gbt
