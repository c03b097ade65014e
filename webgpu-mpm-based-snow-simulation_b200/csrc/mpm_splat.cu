// mpm_splat.cu -- the particle splats the reference's renderers consume,
// into headless device buffers:
//   grid mass   calculateGridMass (src/lib/gpu/volumetric/calculateGridMass.wgsl:8-51):
//               linear-spline splat of particle mass onto the simulation grid,
//               u32 fixed point, for the volumetric ray march;
//   MC density  calculateDensity (src/lib/gpu/marchingCubes/mcDensity.cs.wgsl:14-63):
//               the same splat onto the marching-cubes density grid (half the
//               simulation resolution by default, GpuMarchingCubesBufferManager.ts:44-48),
//               with floor() instead of truncation for the base cell.
// One thread per particle, eight u32 adds, summed per warp first where its
// particles share cells; unsigned addition commutes, so every cell equals the
// reference's total in any order.  Arithmetic follows
// the WGSL expressions operation by operation (no contraction; the kernels are
// compiled with -fmad=false): cellSize = range / res (formed on the host),
// posCell = (pos - min) / cellSize, weight = (wx * wy) * wz, contribution = u32((mass * weight) * scale),
// f32 -> u32 truncating and saturating.
#include <cuda_runtime.h>

#include "mpm_engine.cuh"
#include "mpm_math.cuh"
#include "mpm_splat.cuh"

namespace mpm {

__device__ __forceinline__ uint32_t f2u(float x) { return __float2uint_rz(x); }

constexpr uint32_t NO_CELL = 0xFFFFFFFFu;

// Warp-aggregated add: lanes holding the same cell sum their contributions
// first (u32 addition commutes and wraps, so the cell total is unchanged) and
// one lane adds the sum.  Every lane of the warp calls it; lanes with nothing
// to add pass NO_CELL.
__device__ __forceinline__ void agg_add(uint32_t* out, uint32_t cell, uint32_t v) {
    const uint32_t peers = __match_any_sync(0xffffffffu, cell);
    const uint32_t sum = __reduce_add_sync(peers, v);
    if (cell != NO_CELL && (int)(threadIdx.x & 31u) == __ffs(peers) - 1) atomicAdd(out + cell, sum);
}

// KIND 0: calculateGridMass (truncated base cell, u32 coordinates);
// KIND 1: calculateDensity (floor of the base cell, i32 coordinates).
// MODE 0: one atomic add per lane and cell.  Lanes whose particles share their
// base cell share all eight cells: in modes 1 and 2, where a warp holds at most
// SPLAT_GROUPS base cells, each group sums its contributions and one lane adds
// the sums; the other warps add lane by lane (1) or sum cell by cell (2).
constexpr int SPLAT_GROUPS = 8;

// A particle is read from the caller-order records, or from the planes of the
// work state (in tile order, with the caller index beside it).
template <int KIND, int MODE>
__global__ void __launch_bounds__(256) k_splat(SplatArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = i < (a.ids ? a.n : a.count);
    float pos[3] = {0.f, 0.f, 0.f}, mass = 0.f;
    if (valid && a.ids && a.count != a.n) valid = (__ldg(a.ids + i) & ~ID_KEEP) - a.first < a.count;
    if (valid) {
        const float4* rec = a.ids ? a.particles + i : a.particles + (size_t)(a.first + i) * REC_WORDS;
        float4 q0 = __ldg(rec), q1 = __ldg(rec + (a.ids ? (size_t)a.n : 1));
        pos[0] = q0.x; pos[1] = q0.y; pos[2] = q0.z;
        mass = q1.w;
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (pos[k] < a.gmin[k] || pos[k] >= a.gmax[k]) valid = false;
    }
    int start[3] = {0, 0, 0};
    float w[2][3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float pc = div_any(__fsub_rn(pos[k], a.gmin[k]), a.cell[k], a.rcell[k]);
        float center = __fsub_rn(pc, 0.5f);
        float f;
        if (KIND == 0) {
            uint32_t s0 = f2u(center);
            start[k] = (int)s0;
            f = __fsub_rn(center, __uint2float_rn(s0));
        } else {
            start[k] = __float2int_rz(floorf(center));
            f = __fsub_rn(center, __int2float_rn(start[k]));
        }
        w[0][k] = __fsub_rn(1.0f, f);
        w[1][k] = f;
    }
    uint32_t peers = 0u;
    bool first = true, grouped = false;
    if (MODE != 0) {
        const uint32_t key = valid ? (uint32_t)(start[0] + 1) +
                                         (a.res[0] + 2u) * ((uint32_t)(start[1] + 1) +
                                                            (a.res[1] + 2u) * (uint32_t)(start[2] + 1))
                                   : 0xffffffffu;
        peers = __match_any_sync(0xffffffffu, key);
        first = (int)(threadIdx.x & 31u) == __ffs(peers) - 1;
        grouped = __popc(__ballot_sync(0xffffffffu, first)) <= SPLAT_GROUPS;
    }
    const int rx = (int)a.res[0], ry = (int)a.res[1], rz = (int)a.res[2];
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
        for (int y = 0; y < 2; y++)
#pragma unroll
            for (int x = 0; x < 2; x++) {
                bool in;
                uint32_t cell;
                if (KIND == 0) {
                    uint32_t cx = (uint32_t)start[0] + x, cy = (uint32_t)start[1] + y, cz = (uint32_t)start[2] + z;
                    in = cx < a.res[0] && cy < a.res[1] && cz < a.res[2];
                    cell = cx + a.res[0] * (cy + a.res[1] * cz);
                } else {
                    int cx = start[0] + x, cy = start[1] + y, cz = start[2] + z;
                    in = cx >= 0 && cy >= 0 && cz >= 0 && cx < rx && cy < ry && cz < rz;
                    cell = (uint32_t)(cx + cy * rx + cz * (rx * ry));
                }
                const float weight = __fmul_rn(__fmul_rn(w[x][0], w[y][1]), w[z][2]);
                uint32_t v = f2u(__fmul_rn(__fmul_rn(mass, weight), a.scale));
                if (MODE == 2 && !grouped) {
                    agg_add(a.out, valid && in ? cell : NO_CELL, v);
                } else {
                    if (MODE != 0 && grouped) v = __reduce_add_sync(peers, v);
                    if (valid && in && (first || !grouped)) atomicAdd(a.out + cell, v);
                }
            }
}

cudaError_t launch_splat(int kind, SplatArgs a, cudaStream_t s) {
    const uint32_t n = a.ids ? a.n : a.count;
    if (n == 0 || a.count == 0) return cudaSuccess;
    for (int k = 0; k < 3; k++) {
        volatile float c = a.gmax[k] - a.gmin[k];
        c = c / (float)a.res[k];
        a.cell[k] = c;
        a.rcell[k] = div_recip(c);
    }
    uint32_t blocks = (n + 255u) / 256u;
    // Where the cells outnumber the particles, little contends and the match
    // costs more than it saves; else it pays from four lanes per base cell on,
    // and on a grid of far fewer cells the rest is summed cell by cell.
    // 1,000,000 particles in a fifth of the domain's edge, density pass alone,
    // lattice order / tile order / random order.  Grid 32^3: mode 0 387 / 521 / 398
    // us, 1 35 / 69 / 400, 2 without groups 48 / - / 398.  48^3: 210 / 350 / 172,
    // 41 / 59 / 174, 50 / - / 191.  128^3: 30 / 68 / 92, 46 / 70 / 94.  16^3 in
    // random order: mode 2 438 us, 1 675 us.  Up to 16 groups instead of 8:
    // density pass + marching cubes of 1,500,000 particles, 80^3 cells, 110 -> 126 us.
    const uint64_t cells = (uint64_t)a.res[0] * a.res[1] * a.res[2];
    // the keys fit 32 bits
    const bool keys = (a.res[0] + 2ull) * (a.res[1] + 2ull) < 0xffffffffull / (a.res[2] + 2ull);
    const int mode = !keys || cells >= a.count ? 0 : cells * 32u >= a.count ? 1 : 2;
    void (*const k[2][3])(SplatArgs) = {{k_splat<0, 0>, k_splat<0, 1>, k_splat<0, 2>},
                                        {k_splat<1, 0>, k_splat<1, 1>, k_splat<1, 2>}};
    k[kind == 0 ? 0 : 1][mode]<<<blocks, 256, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace mpm
