// mpm_raymarch.cu -- the volumetric renderer's ray march
// (doVolumetricRaymarch, src/lib/gpu/volumetric/volumetricRaymarch.cs.wgsl:118-226)
// into headless device buffers: an RGBA8 image, an f32 depth image and,
// optionally, the f32 colour before quantisation.  The density field is the
// u32 fixed-point mass grid of calculateGridMass (mpm_splat.cu).
//
// A dense sample marches a 64-step shadow ray (:94-108), so a pixel that sees
// snow evaluates some thousand densities, one after the other in the WGSL.
// Here 4 or 16 lanes (RM_LANES) share a pixel and take its samples in turn: density and
// shadow of a sample do not depend on the samples before it, only the
// compositing does, and that runs in order over the lanes' results.  What
// bounds the pass is the arithmetic of one evaluation and the gathers'
// latency.  Three things keep the arithmetic small without changing a result:
//   - empty space: k_rm_bricks marks the 4^3-cell bricks that lie within a
//     brick of a nonzero cell, and their bounds; outside the bounds and in an
//     unmarked brick every density is 0, so the rays step (their positions
//     still advance by the same rounded additions) past them without
//     evaluating;
//   - the divisions by the cell size and volume become a product with a
//     reciprocal and one correction (div_by), which rounds as the quotient
//     does; the division of each cell by a power-of-two fixed-point scale is
//     exact and moves behind the sum;
//   - exp of the small exponents of one step by a shorter polynomial wherever
//     that provably rounds to the same f32 (exp_step3).
// 1280 x 720 over 128^3 cells, mass splat + march: 4.94 -> 0.74 ms a pass.
// Arithmetic otherwise follows the WGSL expressions operation by operation (no
// contraction, the file is compiled with -fmad=false); exp and pow are the
// project's f64 routines rounded once to f32 (mpm_math.cuh); matrix-vector
// products sum the columns in order, ((c0 x + c1 y) + c2 z) + c3 w; normalize
// divides each component by the IEEE square root of the ordered dot product.
// The workgroupBarrier() calls of the WGSL order nothing here (no shared
// memory) and are left out.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <cuda_runtime.h>

#include "mpm_engine.cuh"
#include "mpm_math.cuh"

namespace mpm {

namespace rm {

constexpr float EXTINCTION = 724.0f;
constexpr float STEP = 0.025f;
constexpr uint32_t N_STEPS = 256u, N_SHADOW_STEPS = 64u;
__device__ __forceinline__ float albedo(int k) { return k == 0 ? 0.9f : (k == 1 ? 0.985f : 0.99f); }
// 4 * PI with PI = 3.1415926, evaluated as an abstract-float constant and
// rounded once to f32
constexpr float FOUR_PI = (float)(4.0 * 3.1415926);
// 1 / 2.2, likewise
constexpr float INV_GAMMA = (float)(1.0 / 2.2);

constexpr int BRICK = 4;   // cells per brick edge

// the light: normalised direction (:119-121), 1 / (its step in bricks)
struct Light {
    float dir[3], rst[3];
};

struct Field {
    const uint32_t* mass;
    float lo[3], hi[3];       // bounds of the marked bricks, a cell wider on each side
    const uint8_t* near;      // per brick: 1 when a nonzero cell lies in it or in one of its 26 neighbours
    uint32_t res[3], bricks[3];
    float gmin[3], gmax[3];
    float cell[3], rcell[3];  // gridRange / gridRes, div_recip(cell)
    float volume, rvolume;    // cellSize.x * cellSize.y * cellSize.z, its div_recip
    float scale, rscale;      // fixedPointScale; 2^-k when it is 2^k, else 0
};

// readDensity (volumetricRaymarch.cs.wgsl:16-57) of a point inside the grid.
// PLAIN: cells or their volume at the ends of the f32 range (plain divisions).
template <bool PLAIN>
__device__ __forceinline__ float read_density(const Field& F, const float* p) {
    uint32_t start[3];
    float w[2][3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float gp = PLAIN ? fd(fs(p[k], F.gmin[k]), F.cell[k]) : div_by(fs(p[k], F.gmin[k]), F.cell[k], F.rcell[k]);
        float sp = fs(gp, 0.5f);
        start[k] = __float2uint_rz(sp);   // saturating: negatives give 0
        float f = fs(sp, __uint2float_rn(start[k]));
        w[0][k] = fs(1.0f, f);
        w[1][k] = f;
    }
    // a cell outside the grid adds nothing; adding its zero product is the same
    const bool in1[3] = {start[0] + 1u < F.res[0], start[1] + 1u < F.res[1], start[2] + 1u < F.res[2]};
    const bool in0 = start[0] < F.res[0] && start[1] < F.res[1] && start[2] < F.res[2];
    if (!in0) return 0.0f;
    const uint32_t* base = F.mass + (start[0] + F.res[0] * (start[1] + F.res[1] * start[2]));
    uint32_t m[2][2][2];
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
        for (int y = 0; y < 2; y++)
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const bool in = (x == 0 || in1[0]) && (y == 0 || in1[1]) && (z == 0 || in1[2]);
                m[z][y][x] = in ? __ldg(base + (size_t)(z ? F.res[0] * F.res[1] : 0u) + (y ? F.res[0] : 0u) + x) : 0u;
            }
    float mass = 0.0f;
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
        for (int y = 0; y < 2; y++)
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const float u = __uint2float_rn(m[z][y][x]);
                const float val = F.rscale != 0.0f ? u : fd(u, F.scale);
                mass = fa(mass, fm(val, fm(fm(w[x][0], w[y][1]), w[z][2])));
            }
    if (F.rscale != 0.0f) mass = fm(mass, F.rscale);
    // (a scale that is no power of two may be tiny, and its masses infinite)
    mass = PLAIN || F.rscale == 0.0f ? fd(mass, F.volume) : div_by(mass, F.volume, F.rvolume);
    return fm(mass, 0.00001f);
}

// Whether a ray whose positions stay within `extent` of the origin may skip
// samples by their number.  A ray's positions are sums of up to 256 rounded
// steps, each off by half an ulp of the extent, where the skips below take them
// to lie evenly: together under 265 * 2^-24 * extent, which has to stay under a
// cell (the marks and their bounds leave more than three).  A ray that may not
// drops only the samples that lie in unmarked bricks, each by itself.
__host__ __device__ inline bool may_skip(float reach, float extent) { return extent < reach; }

// Position of a point in bricks (approximately: the marks reach a whole brick
// beyond the cells a density reads, far more than the rounding here).
__device__ __forceinline__ void brick_of(const Field& F, const float* p, float* g, int* b) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        g[k] = (p[k] - F.gmin[k]) * F.rcell[k] * (1.0f / BRICK);
        b[k] = min(max(__float2int_rd(g[k]), 0), (int)F.bricks[k] - 1);
    }
}
__device__ __forceinline__ bool brick_near(const Field& F, const int* b) {
    return __ldg(F.near + ((size_t)b[2] * F.bricks[1] + b[1]) * F.bricks[0] + b[0]) != 0;
}
// Steps that stay inside the brick: rst = 1 / (step in bricks) per axis.
__device__ __forceinline__ int steps_inside(const float* g, const int* b, const float* rst) {
    float n = 1e9f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float far = (float)(rst[k] > 0.0f ? b[k] + 1 : b[k]);
        n = fminf(n, (far - g[k]) * rst[k]);   // rst = +-inf: inf, or NaN on the face (fminf keeps n)
    }
    return (int)fminf(fmaxf(n, 0.0f), 1024.0f);
}

// Parameters t of o + t d between which the ray lies inside the marked bounds
// (t0 > t1: nowhere).  The bounds are a cell wider than the marks, which covers
// the rounding here.
__device__ __forceinline__ void bounds_range(const Field& F, const float* o, const float* d, float& t0, float& t1) {
    t0 = 0.0f;
    t1 = 3e38f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float r = 1.0f / d[k], a = (F.lo[k] - o[k]) * r, b = (F.hi[k] - o[k]) * r;
        if (d[k] != 0.0f) {
            t0 = fmaxf(t0, fminf(a, b));
            t1 = fminf(t1, fmaxf(a, b));
        } else if (o[k] < F.lo[k] || o[k] > F.hi[k]) {
            t1 = -1.0f;
        }
    }
}

// exp(x) rounded once to f32.  For the exponents of one step, -0.2 <= x <= 0,
// the Taylor polynomial of degree 8 is within 1.5e-12 (13,000 units of the f64
// result in [0.81, 1]) of e^x; unless that reaches a midpoint of two f32 values
// (29 discarded bits), it rounds as the full evaluation does.
// The three channels' polynomials run side by side, with one branch: a third of the
// march's warp time was waits for results of fixed latency.  1280 x 720 over 128^3 cells,
// splat + march, 845 -> 769 us a pass (1,343 -> 1,195 alone), 400 x 225 90 -> 68 us.
__device__ __forceinline__ void exp_step3(const float* x, float* o) {
    double p[3], xd[3];
    bool fast = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        xd[k] = (double)x[k];
        p[k] = __fma_rn(1.0 / 40320.0, xd[k], 1.0 / 5040.0);
        fast = fast && x[k] >= -0.2f && x[k] <= 0.0f;
    }
    const double c[7] = {1.0 / 720.0, 1.0 / 120.0, 1.0 / 24.0, 1.0 / 6.0, 0.5, 1.0, 1.0};
#pragma unroll
    for (int i = 0; i < 7; i++)
#pragma unroll
        for (int k = 0; k < 3; k++) p[k] = __fma_rn(p[k], xd[k], c[i]);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int low = (int)((uint32_t)__double2loint(p[k]) & 0x1fffffffu) - 0x10000000;
        fast = fast && (low > 20000 || low < -20000);
        o[k] = __double2float_rn(p[k]);
    }
    if (!fast) {
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            const float r = expf_m(k == 0 ? x[0] : k == 1 ? x[1] : x[2]);
            if (k == 0) o[0] = r; else if (k == 1) o[1] = r; else o[2] = r;
        }
    }
}

// henyeyGreenstein (:59-63)
__device__ __forceinline__ float hg(float c, float g) {
    float g2 = fm(g, g);
    float denom = fs(fa(1.0f, g2), fm(fm(2.0f, g), c));
    return fd(fs(1.0f, g2), fm(FOUR_PI, powf_m(denom, 1.5f)));
}

// raymarchShadow (:94-108); rst: 1 / (step in bricks)
template <bool PLAIN>
__device__ __forceinline__ void shadow(const Field& F, const float* pos, const float* ld, const float* rst, uint32_t time,
                                       float* T) {
    uint32_t h = hash4(__float_as_uint(pos[0]), __float_as_uint(pos[1]), __float_as_uint(pos[2]), time);
    float jitter = fd(__uint2float_rn(h), 4294967296.0f);
    float sp[3], st[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        st[k] = fm(ld[k], STEP);
        sp[k] = fa(pos[k], fm(st[k], jitter));
        T[k] = 1.0f;
    }
    float t0 = 0.0f, t1 = 3e38f;   // the steps between which the ray is inside the marked bounds
    if (!PLAIN) bounds_range(F, sp, st, t0, t1);
    if (!(t0 <= t1)) return;
    int skip = (int)fminf(fmaxf(t0 - 2.0f, 0.0f), 64.0f);   // samples known to be empty
    const uint32_t n = (uint32_t)fminf(fmaxf(t1 + 2.0f, 0.0f), (float)N_SHADOW_STEPS);
    for (uint32_t s = 0; s < n; s++) {
#pragma unroll
        for (int k = 0; k < 3; k++) sp[k] = fa(sp[k], st[k]);
        if (skip > 0) { skip--; continue; }
        // the light's direction is positive in every axis: past the maximum
        // every later sample is outside
        if (sp[0] >= F.gmax[0] || sp[1] >= F.gmax[1] || sp[2] >= F.gmax[2]) break;
        if (sp[0] < F.gmin[0] || sp[1] < F.gmin[1] || sp[2] < F.gmin[2]) continue;
        float g[3];
        int b[3];
        brick_of(F, sp, g, b);
        if (!brick_near(F, b)) { skip = steps_inside(g, b, rst); continue; }
        float d = read_density<PLAIN>(F, sp);
        if (d > 1e-4f) {
            float a = fm(-fm(EXTINCTION, d), STEP);
            const float x[3] = {fm(a, albedo(0)), fm(a, albedo(1)), fm(a, albedo(2))};
            float e[3];
            exp_step3(x, e);
#pragma unroll
            for (int k = 0; k < 3; k++) T[k] = fm(T[k], e[k]);
            if (T[0] < 1e-4f && T[1] < 1e-4f && T[2] < 1e-4f) break;
        }
    }
}

// uniforms.viewProjInvMat * vec4f(x, y, z, 1), divided by w
__device__ __forceinline__ void unproject(const float* M, float x, float y, float z, float* o) {
    float h[4];
#pragma unroll
    for (int r = 0; r < 4; r++) h[r] = fa(fa(fa(fm(M[r], x), fm(M[4 + r], y)), fm(M[8 + r], z)), fm(M[12 + r], 1.0f));
#pragma unroll
    for (int k = 0; k < 3; k++) o[k] = fd(h[k], h[3]);
}

__device__ __forceinline__ float dot3s(const float* a, const float* b) {
    return fa(fa(fm(a[0], b[0]), fm(a[1], b[1])), fm(a[2], b[2]));
}

__device__ __forceinline__ void normalize3(float* v) {
    float l = __fsqrt_rn(dot3s(v, v));
#pragma unroll
    for (int k = 0; k < 3; k++) v[k] = fd(v[k], l);
}

__device__ __forceinline__ uint8_t unorm8(float v) {
    float c = fminf(fmaxf(v, 0.0f), 1.0f);
    return (uint8_t)__float2uint_rn(fm(c, 255.0f));
}

}  // namespace rm

// Marks the bricks around every nonzero cell and keeps the largest and the
// smallest occupied brick per axis (as bricks - b and b + 1).  One thread per
// row of BRICK cells; own[] keeps the rows of one brick from marking its neighbours again.
__global__ void __launch_bounds__(256) k_rm_bricks(const uint32_t* __restrict__ mass, uint3 res, uint3 bricks,
                                                   uint8_t* __restrict__ own, uint8_t* __restrict__ near,
                                                   uint32_t* __restrict__ bounds) {
    using namespace rm;
    const uint32_t bx = blockIdx.x * 32u + (threadIdx.x & 31u);
    if (bx >= bricks.x) return;
    for (uint32_t z = blockIdx.z; z < res.z; z += gridDim.z)
        for (uint32_t y = blockIdx.y * 8u + (threadIdx.x >> 5); y < res.y; y += gridDim.y * 8u) {
            const uint32_t* row = mass + ((size_t)z * res.y + y) * res.x;
            uint32_t any = 0;
#pragma unroll
            for (uint32_t k = 0; k < BRICK; k++)
                if (bx * BRICK + k < res.x) any |= __ldg(row + bx * BRICK + k);
            if (!any) continue;
            const int b[3] = {(int)bx, (int)(y / BRICK), (int)(z / BRICK)};
            uint8_t* o = own + ((size_t)b[2] * bricks.y + b[1]) * bricks.x + b[0];
            if (*(volatile uint8_t*)o) continue;
            *o = 1;
            const uint32_t n[3] = {bricks.x, bricks.y, bricks.z};
#pragma unroll
            for (int k = 0; k < 3; k++) {   // zero when no brick is occupied
                atomicMax(bounds + k, n[k] - (uint32_t)b[k]);
                atomicMax(bounds + 3 + k, (uint32_t)b[k] + 1u);
            }
            for (int dz = -1; dz <= 1; dz++)
                for (int dy = -1; dy <= 1; dy++)
                    for (int dx = -1; dx <= 1; dx++) {
                        const int x = b[0] + dx, yy = b[1] + dy, zz = b[2] + dz;
                        if (x >= 0 && yy >= 0 && zz >= 0 && x < (int)bricks.x && yy < (int)bricks.y &&
                            zz < (int)bricks.z)
                            near[((size_t)zz * bricks.y + yy) * bricks.x + x] = 1;
                    }
        }
}

// The bound of three CTAs (77 registers) is there for what the compiler does
// without it: 80 with or without spills as the arguments' layout happens to fall
// (320 x 180 pixels over 256^3 cells 442 or 560 us).
template <uint32_t RM_LANES, bool PLAIN>
__global__ void __launch_bounds__(256, 3) k_raymarch(RaymarchArgs a, rm::Field F, rm::Light L) {
    using namespace rm;
    // 16 x 16 / RM_LANES pixels per CTA, RM_LANES neighbouring lanes per pixel
    const uint32_t lane = threadIdx.x & 31u, sub = lane % RM_LANES;
    const uint32_t px = threadIdx.x / RM_LANES;
    const uint32_t gx = blockIdx.x * 16u + (px & 15u), gy = blockIdx.y * (16u / RM_LANES) + (px >> 4);
    if (gx >= a.width || gy >= a.height) return;
    const uint32_t group = ((1u << RM_LANES) - 1u) << (lane - sub);   // the pixel's lanes
    const size_t pix = (size_t)gy * a.width + gx;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        // marks reach one brick beyond the occupied ones
        const float first = (float)F.bricks[k] - (float)__ldg(a.bounds + k), last = (float)__ldg(a.bounds + 3 + k);
        F.lo[k] = F.gmin[k] + ((first - 1.0f) * BRICK - 1.0f) * F.cell[k];
        F.hi[k] = F.gmin[k] + ((last + 1.0f) * BRICK + 1.0f) * F.cell[k];
    }

    // calculateViewRay (shaderPrelude/cameraOps.wgsl:6-19)
    float u = fd(__uint2float_rn(gx), __uint2float_rn(a.width));
    float v = fd(__uint2float_rn(gy), __uint2float_rn(a.height));
    float ux = fs(fm(u, 2.0f), 1.0f), uy = fs(fm(fs(1.0f, v), 2.0f), 1.0f);
    float org[3], far_p[3], dir[3];
    unproject(a.inv_vp, ux, uy, 0.0f, org);
    unproject(a.inv_vp, ux, uy, 1.0f, far_p);
#pragma unroll
    for (int k = 0; k < 3; k++) dir[k] = fs(far_p[k], org[k]);
    normalize3(dir);

    const float* ld = L.dir;
    const float lc[3] = {fm(0.95f, 5.0f), fm(0.995f, 5.0f), fm(1.0f, 5.0f)};
    const float amb[3] = {0.0f, 0.1f, 0.2f};

    // aabbIntersectionDistances (:72-87)
    float t_near = -__int_as_float(0x7f800000), t_far = __int_as_float(0x7f800000);
    {
        float t1[3], t2[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float dmin = fd(fs(a.gmin[k], org[k]), dir[k]);
            float dmax = fd(fs(a.gmax[k], org[k]), dir[k]);
            t1[k] = fminf(dmin, dmax);
            t2[k] = fmaxf(dmin, dmax);
        }
        t_near = fmaxf(fmaxf(t1[0], t1[1]), t1[2]);
        t_far = fminf(fminf(t2[0], t2[1]), t2[2]);
    }

    float d_ground = 1e20f;
    bool hit_ground = false;
    if (fabsf(dir[2]) > 1e-4f) {
        float cand = fd(fs(a.gmin[2], org[2]), dir[2]);
        if (cand > 0.0f) {
            float hx = fa(org[0], fm(cand, dir[0])), hy = fa(org[1], fm(cand, dir[1]));
            if (hx >= a.gmin[0] && hy >= a.gmin[1] && hx <= a.gmax[0] && hy <= a.gmax[1]) {
                d_ground = cand;
                hit_ground = true;
            }
        }
    }

    if (!(t_near <= t_far && t_far >= 0.0f)) {
        if (sub != 0u) return;
        reinterpret_cast<uchar4*>(a.rgba)[pix] = make_uchar4(0, 0, 0, 0);
        if (a.color) reinterpret_cast<float4*>(a.color)[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;   // the depth image keeps its previous content, as the reference's texture does
    }

    const float d_start = fmaxf(0.0f, t_near);
    const float d_end = fminf(t_far, d_ground);
    float jitter = fd(__uint2float_rn(hash3(gx, gy, a.time)), 4294967296.0f);
    float cur = fa(d_start, fm(jitter, STEP));

    float T[3] = {1.0f, 1.0f, 1.0f}, col[3] = {0.0f, 0.0f, 0.0f};
    bool depth_written = false;
    float depth = 1e20f;

    // the part of the ray inside the marked bounds, in steps from cur
    const bool fine = may_skip(a.reach, fmaxf(fabsf(org[0]), fmaxf(fabsf(org[1]), fabsf(org[2]))) + cur + (N_STEPS + 1u) * STEP);
    float t0 = 0.0f, t1 = 3e38f;
    if (fine) {
        float o[3], d[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            o[k] = fa(org[k], fm(cur, dir[k]));
            d[k] = fm(dir[k], STEP);
        }
        bounds_range(F, o, d, t0, t1);
    }
    float phase = 0.0f, rst[3] = {0.f, 0.f, 0.f};
    if (t0 <= t1) {
        // the phase function depends only on the ray: evaluated once
        phase = fa(hg(dot3s(dir, ld), -0.5f), hg(dot3s(dir, ld), 0.5f));
#pragma unroll
        for (int k = 0; k < 3; k++) rst[k] = fine ? BRICK * F.cell[k] / (dir[k] * STEP) : 0.0f;   // 1 / (step in bricks); 0: no step is inside
    }
    const uint32_t n = t0 <= t1 ? (uint32_t)fminf(fmaxf(t1 + 2.0f, 0.0f), (float)N_STEPS) : 0u;
    uint32_t i = (uint32_t)fminf(fmaxf(t0 - 2.0f, 0.0f), (float)N_STEPS);   // samples before it are empty
    for (uint32_t k = 0; k < i && i < n; k++) cur = fa(cur, STEP);
    // the pixel's lanes hold the same i, cur, T, col; lane `sub` takes sample i + sub
    while (i < n && cur < d_end && !(T[0] < 0.01f && T[1] < 0.01f && T[2] < 0.01f)) {
        float pos[3], g[3];
        int b[3];
#pragma unroll
        for (int k = 0; k < 3; k++) pos[k] = fa(org[k], fm(cur, dir[k]));
        const bool in0 = pos[0] >= F.gmin[0] && pos[1] >= F.gmin[1] && pos[2] >= F.gmin[2] && pos[0] < F.gmax[0] &&
                         pos[1] < F.gmax[1] && pos[2] < F.gmax[2];
        brick_of(F, pos, g, b);
        if (!in0 || !brick_near(F, b)) {
            const uint32_t skip = in0 ? (uint32_t)steps_inside(g, b, rst) + 1u : 1u;
            for (uint32_t k = 0; k < skip && i < n; k++, i++) cur = fa(cur, STEP);
            continue;
        }
        float c = cur;
        for (uint32_t k = 0; k < sub; k++) c = fa(c, STEP);
        float density = 0.0f;
        if (i + sub < n && c < d_end) {
#pragma unroll
            for (int k = 0; k < 3; k++) pos[k] = fa(org[k], fm(c, dir[k]));
            if (pos[0] >= F.gmin[0] && pos[1] >= F.gmin[1] && pos[2] >= F.gmin[2] && pos[0] < F.gmax[0] &&
                pos[1] < F.gmax[1] && pos[2] < F.gmax[2])
                density = read_density<PLAIN>(F, pos);
        }
        const bool dense = density > 0.001f;
        float laf[3] = {0.f, 0.f, 0.f}, stT[3] = {1.f, 1.f, 1.f};
        if (dense) {
            float ext = fm(EXTINCTION, density);
            float a_ext = fm(-ext, STEP);
            float sh[3];
            shadow<PLAIN>(F, pos, ld, L.rst, a.time, sh);
            float inv_ext = fmaxf(ext, 1e-4f);
            const float x[3] = {fm(a_ext, albedo(0)), fm(a_ext, albedo(1)), fm(a_ext, albedo(2))};
            exp_step3(x, stT);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                float scat = fm(ext, albedo(k));
                float light = fa(amb[k], fm(fm(lc[k], phase), sh[k]));
                laf[k] = fd(fm(fm(light, scat), fs(1.0f, stT[k])), inv_ext);
            }
        }
        // composite the samples in order; a sample past the end is not dense
        const uint32_t hits = __ballot_sync(group, dense);
        for (uint32_t j = 0; j < RM_LANES; j++) {
            const int src = (int)(lane - sub + j);
            if (!(hits >> src & 1u)) continue;
            if (T[0] < 0.01f && T[1] < 0.01f && T[2] < 0.01f) break;
            const float cj = __shfl_sync(group, c, src);
            if (!depth_written) {
                depth = cj;
                depth_written = true;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                col[k] = fa(col[k], fm(T[k], __shfl_sync(group, laf[k], src)));
                T[k] = fm(T[k], __shfl_sync(group, stT[k], src));
            }
        }
        cur = fa(__shfl_sync(group, c, (int)(lane - sub + RM_LANES - 1u)), STEP);
        i += RM_LANES;
    }

    if (hit_ground && (T[0] > 0.01f || T[1] > 0.01f || T[2] > 0.01f)) {
        float pos[3], sh[3];
#pragma unroll
        for (int k = 0; k < 3; k++) pos[k] = fa(org[k], fm(d_ground, dir[k]));
        shadow<PLAIN>(F, pos, ld, L.rst, a.time, sh);
        float lz = fmaxf(0.0f, ld[2]);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float gcol = fa(amb[k], fm(0.05f, fm(fm(lc[k], sh[k]), lz)));
            col[k] = fa(col[k], fm(T[k], gcol));
            T[k] = 0.0f;
        }
        if (!depth_written) depth = d_ground;
    }

    // lane k < 3 of the pixel takes colour channel k
    const float alpha = fs(1.0f, fmaxf(T[0], fmaxf(T[1], T[2])));
    const float ch = sub == 0u ? col[0] : (sub == 1u ? col[1] : col[2]);
    const float oc = sub < 3u ? fm(powf_m(ch, INV_GAMMA), alpha) : 0.0f;
    const float o1 = __shfl_sync(group, oc, (int)(lane - sub + 1u)), o2 = __shfl_sync(group, oc, (int)(lane - sub + 2u));
    if (sub != 0u) return;
    const float o[4] = {oc, o1, o2, fm(1.0f, alpha)};
    reinterpret_cast<uchar4*>(a.rgba)[pix] = make_uchar4(unorm8(o[0]), unorm8(o[1]), unorm8(o[2]), unorm8(o[3]));
    if (a.color) reinterpret_cast<float4*>(a.color)[pix] = make_float4(o[0], o[1], o[2], o[3]);
    a.depth[pix] = depth;
}

size_t raymarch_workspace(const uint32_t* res) {
    size_t n = 1;
    for (int k = 0; k < 3; k++) n *= (res[k] + rm::BRICK - 1u) / rm::BRICK;
    return 32 + 2 * n;
}

cudaError_t launch_raymarch(RaymarchArgs a, uint8_t* ws, cudaStream_t s) {
    if (a.width == 0 || a.height == 0) return cudaSuccess;
    const uint3 res = make_uint3(a.res[0], a.res[1], a.res[2]);
    const uint3 br = make_uint3((res.x + rm::BRICK - 1u) / rm::BRICK, (res.y + rm::BRICK - 1u) / rm::BRICK,
                                (res.z + rm::BRICK - 1u) / rm::BRICK);
    const size_t n = (raymarch_workspace(a.res) - 32) / 2;
    // everything the pixels share, one IEEE f32 operation at a time
    rm::Field F{};
    rm::Light L{};
    volatile float v;
    for (int k = 0; k < 3; k++) {
        F.res[k] = a.res[k];
        F.bricks[k] = (a.res[k] + rm::BRICK - 1u) / rm::BRICK;
        F.gmin[k] = a.gmin[k];
        F.gmax[k] = a.gmax[k];
        v = a.gmax[k] - a.gmin[k];
        v = v / (float)a.res[k];
        F.cell[k] = v;
        F.rcell[k] = div_recip(v);
    }
    v = F.cell[0] * F.cell[1];
    v = v * F.cell[2];
    F.volume = v;
    F.rvolume = div_recip(v);
    // plain: every brick marked, no skips
    const bool plain = F.rcell[0] == 0.0f || F.rcell[1] == 0.0f || F.rcell[2] == 0.0f || F.rvolume == 0.0f;
    a.reach = plain ? 0.0f : std::min(F.cell[0], std::min(F.cell[1], F.cell[2])) * (16777216.0f / 265.0f);
    // shadow rays start inside the grid
    float extent = 0.0f;
    for (int k = 0; k < 3; k++) extent = std::max(extent, std::max(std::fabs(a.gmin[k]), std::fabs(a.gmax[k])));
    const bool shadow_skips = rm::may_skip(a.reach, extent + (rm::N_SHADOW_STEPS + 1u) * rm::STEP);
    F.scale = a.scale;
    // 2^-k when the scale is 2^k, k <= 46 (then u / scale is exact, and no
    // product with a weight underflows), else 0
    uint32_t bits;
    memcpy(&bits, &a.scale, 4);
    const int ex = (int)(bits >> 23);
    F.rscale = (bits & 0x7fffffu) == 0u && ex >= 127 && ex <= 127 + 46 ? 1.0f / a.scale : 0.0f;
    const float l0[3] = {0.2f, 0.18f, 0.9f};
    volatile float xx = l0[0] * l0[0], yy = l0[1] * l0[1], zz = l0[2] * l0[2];
    v = xx + yy;
    v = v + zz;
    volatile float len = std::sqrt((float)v);
    for (int k = 0; k < 3; k++) {
        v = l0[k] / len;
        L.dir[k] = v;
        L.rst[k] = shadow_skips ? rm::BRICK * F.cell[k] / (L.dir[k] * rm::STEP) : 0.0f;
    }
    a.bounds = reinterpret_cast<uint32_t*>(ws);
    uint8_t* own = ws + 32;
    F.mass = a.mass;
    F.near = own + n;
    cudaError_t e = cudaMemsetAsync(ws, plain ? 1 : 0, 32 + 2 * n, s);
    if (e != cudaSuccess) return e;
    if (!plain) k_rm_bricks<<<dim3((br.x + 31u) / 32u, std::min((res.y + 7u) / 8u, 65535u), std::min(res.z, 65535u)), 256, 0, s>>>(
        a.mass, res, br, own, own + n, reinterpret_cast<uint32_t*>(ws));
    const uint64_t pixels = (uint64_t)a.width * a.height;
    // Lanes per pixel.  The dense pixels of an image are too few to fill the
    // GPU with a thread each, and their chains of evaluations then set the time
    // (1280 x 720, one thread per pixel: 1.32 ms a pass back to back over three
    // scenes, 3.5 ms alone; 4 lanes 0.85 / 1.36); more lanes repeat the empty
    // pixels' setup.  4 against 16 lanes, 300,000 particles: 360 x 200 411 /
    // 1163 -> 195 / 479 us, 640 x 360 419 / 1136 -> 432 / 614, 800 x 450
    // 454 / 1194 -> 645 / 750 (8 lanes: 252 / 674, 426 / 741, 622 / 871).
    const bool general = plain || !shadow_skips;
    const uint32_t lanes = !general && pixels < 250000u ? 16u : 4u;
    const uint32_t rows = 16u / lanes;
    const dim3 grid((a.width + 15u) / 16u, (a.height + rows - 1u) / rows);
    if (general) k_raymarch<4, true><<<grid, 256, 0, s>>>(a, F, L);
    else if (lanes == 4u) k_raymarch<4, false><<<grid, 256, 0, s>>>(a, F, L);
    else k_raymarch<16, false><<<grid, 256, 0, s>>>(a, F, L);
    return cudaGetLastError();
}

}  // namespace mpm
