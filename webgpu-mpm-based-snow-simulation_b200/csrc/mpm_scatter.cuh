// mpm_scatter.cuh -- arguments of the particle scatter (mpm_scatter.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace mpm {

struct ScatterArgs {
    float4* particles;         // n records (12 float4 each)
    uint32_t n;
    uint32_t n_tris;
    float mmin[3], mmax[3];    // meshMinCoords, meshMaxCoords
    // set by launch_scatter, in the workspace
    const float4* verts;       // triangle soup, 3 vertices per triangle (xyz, pad)
    float4* tris;              // 3 float4 per triangle (sc_record)
    uint32_t* range;           // bins each triangle covers: y lo, hi, z lo, hi (8 bits each); lo > hi: none
    uint32_t* count;           // bins^2
    uint32_t* start;           // bins^2 + 1: list range of each bin
    uint32_t* list;            // cap triangle indices
    unsigned long long* large; // bins covered by the triangles of more than SC_LARGE bins
    uint32_t bins, cap;
    float blo[2], binv[2];     // bin grid origin (y, z) and bins per unit
};

// Room for the bins' lists: SC_LARGE entries per triangle, and sc_budget for
// those of the triangles in more bins than that.
constexpr uint32_t SC_LARGE = 16;
inline __host__ __device__ uint32_t sc_budget(uint32_t n_tris) {
    return 32u * (n_tris < (1u << 26) ? n_tris : (1u << 26)) + 16384u;
}
inline uint32_t scatter_cap(uint32_t n_tris) {
    return SC_LARGE * (n_tris < (1u << 26) ? n_tris : (1u << 26)) + sc_budget(n_tris);
}
size_t scatter_workspace(uint32_t n_tris);
// Copies the host triangle soup (n_tris * 3 vertices of 4 floats) into the
// workspace and fills the records, all enqueued on s.
cudaError_t launch_scatter(ScatterArgs a, const float* host_verts, char* ws, cudaStream_t s);

}  // namespace mpm
