// mpm_splat.cuh -- arguments of the renderers' particle splats (mpm_splat.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace mpm {

struct SplatArgs {
    const float4* particles;   // caller-order records, or the work state's planes when ids is given
    const uint32_t* ids;       // nullptr, or the caller index of each of the n work slots
    uint32_t n;
    uint32_t first, count;     // the scene's records
    float gmin[3], gmax[3];
    uint32_t res[3];           // splat grid resolution
    float scale;               // fixedPointScale
    uint32_t* out;             // res[0] * res[1] * res[2] u32
    float cell[3], rcell[3];   // set by launch_splat: cell size, div_recip(cell)
};

cudaError_t launch_splat(int kind, SplatArgs a, cudaStream_t s);

}  // namespace mpm
