// generate_triangular_surface over the engine's C ABI
// (reference: marching_cubes.cu:159-237).
#include "cuphoto/marching_cubes.cuh"

#include <cstdio>

namespace cuphoto {

namespace {

// The mesh's device buffers, allocated by gbt_extract_mesh_sized's callback.
struct MeshBuffers {
    float* verts = nullptr;
    float* normals = nullptr;
    int32_t* tris = nullptr;
    bool with_normals = false;

    ~MeshBuffers() {
        cudaFree(verts);
        cudaFree(normals);
        cudaFree(tris);
    }
    static int alloc(void* ctx, int64_t n_verts, int64_t n_tris, float** verts, float** normals, int32_t** tris) {
        MeshBuffers* b = static_cast<MeshBuffers*>(ctx);
        if (n_tris == 0) return 0;
        const size_t bytes = (size_t)n_verts * 3 * sizeof(float);
        if (cudaMalloc(&b->verts, bytes) != cudaSuccess ||
            (b->with_normals && cudaMalloc(&b->normals, bytes) != cudaSuccess) ||
            cudaMalloc(&b->tris, (size_t)n_tris * 3 * sizeof(int32_t)) != cudaSuccess) {
            cudaGetLastError();
            return 1;
        }
        *verts = b->verts;
        *normals = b->normals;
        *tris = b->tris;
        return 0;
    }
};

}  // namespace

void generate_triangular_surface(const TSDFVolume& tsdf_volume, std::vector<float3>& vertices,
                                 std::vector<int3>& triangles) {
    gbt_volume* vol = tsdf_volume.engine();
    if (!vol) {
        std::fprintf(stderr, "[cuda]   generate_triangular_surface() -- volume was not allocated\n");
        return;
    }
    MeshBuffers b;
    const int64_t base = (int64_t)vertices.size();
    int64_t nv = 0, n = 0;
    if (gbt_extract_mesh_sized(vol, 0, MeshBuffers::alloc, &b, base, &nv, &n, nullptr) != GBT_OK) {
        std::fprintf(stderr, "[cuda]   generate_triangular_surface() -- %s\n", gbt_last_error());
        return;
    }
    if (n == 0) return;
    const size_t v0 = vertices.size(), t0 = triangles.size();
    vertices.resize(v0 + (size_t)nv);
    triangles.resize(t0 + (size_t)n);
    cudaMemcpy(vertices.data() + v0, b.verts, (size_t)nv * 3 * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(triangles.data() + t0, b.tris, (size_t)n * 3 * sizeof(int32_t), cudaMemcpyDeviceToHost);
}

bool generate_indexed_surface(const TSDFVolume& tsdf_volume, std::vector<float3>& vertices,
                              std::vector<float3>& normals, std::vector<int3>& triangles) {
    gbt_volume* vol = tsdf_volume.engine();
    if (!vol) {
        std::fprintf(stderr, "[cuda]   generate_indexed_surface() -- volume was not allocated\n");
        return false;
    }
    MeshBuffers b;
    b.with_normals = true;
    const int64_t base = (int64_t)vertices.size();
    int64_t nv = 0, nt = 0;
    if (gbt_extract_mesh_sized(vol, 1, MeshBuffers::alloc, &b, base, &nv, &nt, nullptr) != GBT_OK) {
        std::fprintf(stderr, "[cuda]   generate_indexed_surface() -- %s\n", gbt_last_error());
        return false;
    }
    normals.resize(vertices.size());
    if (nt == 0) return true;
    const size_t v0 = vertices.size(), t0 = triangles.size();
    vertices.resize(v0 + (size_t)nv);
    normals.resize(v0 + (size_t)nv);
    triangles.resize(t0 + (size_t)nt);
    cudaMemcpy(vertices.data() + v0, b.verts, (size_t)nv * 3 * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(normals.data() + v0, b.normals, (size_t)nv * 3 * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(triangles.data() + t0, b.tris, (size_t)nt * 3 * sizeof(int32_t), cudaMemcpyDeviceToHost);
    return true;
}

}  // namespace cuphoto
