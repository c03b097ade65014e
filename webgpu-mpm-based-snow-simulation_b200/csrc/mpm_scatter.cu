// mpm_scatter.cu -- particle initialisation: scatterParticles
// (src/lib/gpu/particleInitialize/particleScatter.cs.wgsl:47-84).  Each
// particle draws candidates uniformly in the mesh's bounding box
// (uniforms.meshMinCoords / meshMaxCoords) from its own hash stream until one
// lies inside the closed triangle mesh (even-odd count of Moller-Trumbore
// hits along +x, triangleOps.wgsl), at most 512 attempts, then jitters it by
// three fBm values (randomNumberGenerators.wgsl:57-94) and draws its mass.
//
// B200 form: the rays all run along +x, so only triangles whose projection on
// the (y, z) plane covers a candidate can be hit.  Each call bins the triangles
// into a G x G grid over that plane (k_sc_prep counts, k_sc_scan places,
// k_sc_fill lists) and one thread per particle tests a candidate against its
// cell's list only; what a triangle contributes to every ray (edges, 1 / det)
// is formed once per triangle.  Each kept triangle gives the hit test of the
// sequential loop, operation by operation, the dropped ones provably give "no
// hit", and the parity does not depend on the order, so the result equals the
// reference's loop over all triangles.  Testing every triangle against every
// candidate, with an IEEE division each, took 13.5 ms for 65,536 particles in
// 5,120 triangles; with the bins the call takes 0.18 ms, much of it the copy
// of the vertices.  Arithmetic: the step's f32 helpers (dot and
// cross with the canonical fused order), IEEE division, mix(a, b, t) =
// a (1 - t) + b t unfused, fract(x) = x - floor(x).
#include <cuda_runtime.h>

#include "mpm_math.cuh"
#include "mpm_scatter.cuh"

namespace mpm {


constexpr int SCATTER_BS = 128;
constexpr uint32_t SC_CHUNK = 256;
constexpr uint32_t SCATTER_MAX_ATTEMPTS = 512u;

__device__ __forceinline__ float u32_unit(uint32_t h) { return fd(__uint2float_rn(h), 4294967296.0f); }
__device__ __forceinline__ float mixf(float a, float b, float t) { return fa(fm(a, fs(1.0f, t)), fm(b, t)); }

__device__ __forceinline__ float rand_float(uint32_t& seed) {
    seed = hash1(seed);
    return u32_unit(seed);
}

// Cell of coordinate k (0: y, 1: z) of the bin grid.  Monotone in v, so a value
// between two others lies in a cell between theirs; NaN gives cell 0.
__device__ __forceinline__ int sc_cell(const ScatterArgs& a, int k, float v) {
    const int c = __float2int_rd(fm(fs(v, a.blo[k]), a.binv[k]));
    return min(max(c, 0), (int)a.bins - 1);
}

// Ray record of triangle t: vertex 0 and 1 / det, edges e1 = v1 - v0 and
// e2 = v2 - v0.  With the ray along +x, cross(dir, e2) = (0, -e2.z, e2.y).
// False for a triangle no ray can hit: |det| under the test's epsilon, or a
// vertex or det that is not finite (the hit test then ends in a comparison
// with NaN or with 0, which fails).
__device__ __forceinline__ bool sc_record(const ScatterArgs& a, uint32_t t, float4* r) {
    const float eps = 1e-6f;
    const float4 v0 = __ldg(a.verts + (size_t)t * 3), v1 = __ldg(a.verts + (size_t)t * 3 + 1),
                 v2 = __ldg(a.verts + (size_t)t * 3 + 2);
    const float e1[3] = {fs(v1.x, v0.x), fs(v1.y, v0.y), fs(v1.z, v0.z)};
    const float e2[3] = {fs(v2.x, v0.x), fs(v2.y, v0.y), fs(v2.z, v0.z)};
    const float det = ff(e1[2], e2[1], fm(e1[1], -e2[2]));
    r[0] = make_float4(v0.x, v0.y, v0.z, fd(1.0f, det));
    r[1] = make_float4(e1[0], e1[1], e1[2], e2[0]);
    r[2] = make_float4(e2[1], e2[2], det, 0.f);
    const float all = v0.x * 0.f + v0.y * 0.f + v0.z * 0.f + e1[0] * 0.f + e1[1] * 0.f + e1[2] * 0.f + e2[0] * 0.f +
                      e2[1] * 0.f + e2[2] * 0.f + det * 0.f;
    return all == 0.f && !(fabsf(det) < eps);
}

// rayIntersectsTriangle (triangleOps.wgsl), ray direction +x, from a record
__device__ __forceinline__ bool ray_x_hits(const float* o, const float4& r0, const float4& r1, const float4& r2) {
    const float eps = 1e-6f;
    const float inv = r0.w, e1[3] = {r1.x, r1.y, r1.z}, e2[3] = {r1.w, r2.x, r2.y};
    const float ov[3] = {fs(o[0], r0.x), fs(o[1], r0.y), fs(o[2], r0.z)};
    const float b0 = fm(ff(ov[2], e2[1], fm(ov[1], -e2[2])), inv);
    if (b0 < 0.0f || 1.0f < b0) return false;
    float ove1[3];
    cross3(ov, e1, ove1);
    const float b1 = fm(ff(0.0f, ove1[2], ff(0.0f, ove1[1], ove1[0])), inv);   // dot(dir, ove1)
    if (b1 < 0.0f || 1.0f < b1 || fa(b0, b1) > 1.0f) return false;
    return fm(dot3(e2, ove1), inv) > eps;
}

// Bins a triangle can be hit from.  A hit needs computed barycentrics b0, b1
// in [0, 1] with b0 + b1 <= 1; rounding moves them by at most tau = 16 ulp
// ((D max(S1, S2) + S1 S2) / |det| + 1), where D bounds |candidate - v0| and
// S1, S2 the edges in the (y, z) plane, so the candidate lies within
// 3 tau (|e1| + |e2|) of the projected triangle (and half an ulp of its
// coordinates).  Slivers, whose tau is large, cover many bins.
__device__ __forceinline__ void sc_bins(const ScatterArgs& a, const float4* r, int* lo, int* hi) {
    const float v0[2] = {r[0].y, r[0].z}, e1[2] = {r[1].y, r[1].z}, e2[2] = {r[2].x, r[2].y};
    float D = 0.f;
#pragma unroll
    for (int k = 0; k < 2; k++) D += fmaxf(fabsf(a.mmin[k + 1] - v0[k]), fabsf(a.mmax[k + 1] - v0[k]));
    const float S1 = fabsf(e1[0]) + fabsf(e1[1]), S2 = fabsf(e2[0]) + fabsf(e2[1]);
    const float tau = 1e-6f * ((D * fmaxf(S1, S2) + S1 * S2) / fabsf(r[2].z) + 1.0f);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float m = 3.0f * tau * (fabsf(e1[k]) + fabsf(e2[k])) + 1e-6f * (fabsf(v0[k]) + fabsf(e1[k]) + fabsf(e2[k]) + D);
        const float l = v0[k] + fminf(0.f, fminf(e1[k], e2[k])) - m, h = v0[k] + fmaxf(0.f, fmaxf(e1[k], e2[k])) + m;
        const bool ok = l <= h;   // false for NaN: every bin
        lo[k] = ok ? sc_cell(a, k, l) : 0;
        hi[k] = ok ? sc_cell(a, k, h) : (int)a.bins - 1;
    }
}

// One warp per triangle: its record, and one count in each bin it covers.  Once
// the triangles of many bins have used up their share of the lists, these
// cannot fit and nothing more is counted (72,000 triangles over the whole mesh
// box: 1.2e9 counts took 60 of 145 ms).
__global__ void __launch_bounds__(128) k_sc_prep(ScatterArgs a) {
    const uint32_t t = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (t >= a.n_tris) return;
    float4 r[3];
    int lo[2] = {1, 1}, hi[2] = {0, 0};
    if (sc_record(a, t, r)) {
        sc_bins(a, r, lo, hi);
        r[2].w = 1.f;
    }
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 3; q++) a.tris[(size_t)t * 3 + q] = r[q];
        a.range[t] = (uint32_t)lo[0] | (uint32_t)hi[0] << 8 | (uint32_t)lo[1] << 16 | (uint32_t)hi[1] << 24;
    }
    const int ny = hi[0] - lo[0] + 1, n = ny * (hi[1] - lo[1] + 1);
    if (n > (int)SC_LARGE) {
        unsigned long long before = 0;
        if (lane == 0) before = atomicAdd(a.large, (unsigned long long)n);
        before = __shfl_sync(0xffffffffu, before, 0);
        if (before + (unsigned long long)n > sc_budget(a.n_tris)) return;
    }
    for (int i = (int)lane; i < n; i += 32)
        atomicAdd(a.count + (uint32_t)(lo[1] + i / ny) * a.bins + (uint32_t)(lo[0] + i % ny), 1u);
}

// Exclusive scan of the bin counts by one CTA: start[0 .. bins^2]; the counts
// become the bins' fill cursors.  A triangle may lie in every bin, so a total
// may pass 32 bits: it is summed in 64 bits and kept saturated.  All ones, which
// no cap reaches, where the lists do not fit (the starts are then not read).
__global__ void __launch_bounds__(1024) k_sc_scan(ScatterArgs a) {
    __shared__ unsigned long long wsum[32];
    const uint32_t n = a.bins * a.bins, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (uint32_t b0 = 0; b0 < n; b0 += 1024u) {
        const uint32_t i = b0 + threadIdx.x, v = i < n ? a.count[i] : 0u;
        unsigned long long x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) x += y;
        }
        if (lane == 31u) wsum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned long long w = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
                if ((int)lane >= o) w += y;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        const uint32_t ex = (uint32_t)(carry + (warp ? wsum[warp - 1u] : 0ull) + x - v);
        carry += wsum[31];
        if (i < n) {
            a.start[i] = ex;
            a.count[i] = ex;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        a.start[n] = carry <= a.cap && *a.large <= sc_budget(a.n_tris) ? (uint32_t)carry : 0xffffffffu;
}

// One warp per triangle: its index into the list of each bin it covers.  When
// the lists do not fit (many large or sliver triangles), the particles test
// every triangle instead.
__global__ void __launch_bounds__(128) k_sc_fill(ScatterArgs a) {
    const uint32_t t = blockIdx.x * 4u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (t >= a.n_tris || a.start[a.bins * a.bins] > a.cap) return;
    const uint32_t g = a.range[t];
    const int lo0 = (int)(g & 255u), ny = (int)(g >> 8 & 255u) - lo0 + 1, lo1 = (int)(g >> 16 & 255u);
    const int n = ny * ((int)(g >> 24) - lo1 + 1);
    for (int i = (int)lane; i < n; i += 32)
        a.list[atomicAdd(a.count + (uint32_t)(lo1 + i / ny) * a.bins + (uint32_t)(lo0 + i % ny), 1u)] = t;
}

__device__ __forceinline__ float noise3(float x0, float x1, float x2) {
    float x[3] = {x0, x1, x2}, f[3], u[3];
    uint32_t n[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float p = floorf(x[k]);
        f[k] = fs(x[k], p);
        u[k] = fm(fm(f[k], f[k]), fs(3.0f, fm(2.0f, f[k])));
        n[k] = (uint32_t)__float2int_rz(p);
    }
    float c[8];
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = u32_unit(hash3(n[0] + (i & 1), n[1] + ((i >> 1) & 1), n[2] + (i >> 2)));
    return mixf(mixf(mixf(c[0], c[1], u[0]), mixf(c[2], c[3], u[0]), u[1]),
                mixf(mixf(c[4], c[5], u[0]), mixf(c[6], c[7], u[0]), u[1]), u[2]);
}

__device__ __forceinline__ float fbm3(float x0, float x1, float x2) {
    float v = 0.0f, a = 0.5f;
#pragma unroll 1
    for (int i = 0; i < 6; i++) {
        v = fa(v, fm(a, noise3(x0, x1, x2)));
        x0 = fm(x0, 2.0f);
        x1 = fm(x1, 2.0f);
        x2 = fm(x2, 2.0f);
        a = fm(a, 0.5f);
    }
    return v;
}

// Where the lists do not fit, the CTA's candidates are tested against every
// triangle, SC_CHUNK records at a time through shared memory.
__global__ void __launch_bounds__(SCATTER_BS) k_scatter(ScatterArgs a) {
    __shared__ float4 tri[SC_CHUNK * 3];
    const uint32_t i = blockIdx.x * SCATTER_BS + threadIdx.x;
    uint32_t seed = hash4(i, 100u, 200u, 300u);
    float cand[3] = {0.f, 0.f, 0.f};
    if (a.start[a.bins * a.bins] <= a.cap) {
        if (i >= a.n) return;
        for (uint32_t attempt = 0; attempt < SCATTER_MAX_ATTEMPTS; attempt++) {
#pragma unroll
            for (int k = 0; k < 3; k++) cand[k] = mixf(a.mmin[k], a.mmax[k], rand_float(seed));
            const uint32_t c = (uint32_t)sc_cell(a, 1, cand[2]) * a.bins + (uint32_t)sc_cell(a, 0, cand[1]);
            const uint32_t end = __ldg(a.start + c + 1);
            bool inside = false;
            for (uint32_t e = __ldg(a.start + c); e < end; e++) {
                const float4* r = a.tris + (size_t)__ldg(a.list + e) * 3;
                if (ray_x_hits(cand, __ldg(r), __ldg(r + 1), __ldg(r + 2))) inside = !inside;
            }
            if (inside) break;
        }
    } else {
        bool done = i >= a.n;
        for (uint32_t attempt = 0; attempt < SCATTER_MAX_ATTEMPTS; attempt++) {
            if (__syncthreads_and(done ? 1 : 0)) break;
            if (!done) {
#pragma unroll
                for (int k = 0; k < 3; k++) cand[k] = mixf(a.mmin[k], a.mmax[k], rand_float(seed));
            }
            bool inside = false;
            for (uint32_t t0 = 0; t0 < a.n_tris; t0 += SC_CHUNK) {
                const uint32_t nt = min(SC_CHUNK, a.n_tris - t0);
                __syncthreads();
                for (uint32_t k = threadIdx.x; k < nt * 3; k += SCATTER_BS) tri[k] = __ldg(a.tris + (size_t)t0 * 3 + k);
                __syncthreads();
                if (!done)
                    for (uint32_t t = 0; t < nt; t++) {
                        const float4 r2 = tri[3 * t + 2];
                        if (r2.w != 0.f && ray_x_hits(cand, tri[3 * t], tri[3 * t + 1], r2)) inside = !inside;
                    }
            }
            done = done || inside;
        }
        if (i >= a.n) return;
    }
    const float freq = 4.0f, scale = 0.1f;
    float x[3] = {fm(cand[0], freq), fm(cand[1], freq), fm(cand[2], freq)};
    float d0 = fbm3(x[0], x[1], x[2]);
    float d1 = fbm3(fa(x[0], 100.0f), fa(x[1], 200.0f), fa(x[2], 300.0f));
    float d2 = fbm3(fa(x[0], -300.0f), fa(x[1], -200.0f), fa(x[2], -100.0f));
    float pos[3] = {fa(cand[0], fm(fs(d0, 0.5f), scale)), fa(cand[1], fm(fs(d1, 0.5f), scale)),
                    fa(cand[2], fm(fs(d2, 0.5f), scale))};
    float m1 = u32_unit(hash1(i));
    float4* rec = a.particles + (size_t)i * 12;
    rec[0] = make_float4(pos[0], pos[1], pos[2], 1.0f);
    rec[1] = make_float4(0.f, 0.f, 0.f, fm(m1, m1));
    rec[2] = make_float4(1.f, 0.f, 0.f, 0.f);
    rec[3] = make_float4(0.f, 1.f, 0.f, 0.f);
    rec[4] = make_float4(0.f, 0.f, 1.f, 0.f);
    rec[5] = make_float4(1.f, 0.f, 0.f, 0.f);
    rec[6] = make_float4(0.f, 1.f, 0.f, 0.f);
    rec[7] = make_float4(0.f, 0.f, 1.f, 0.f);
    for (int q = 8; q < 12; q++) rec[q] = make_float4(0.f, 0.f, 0.f, 0.f);
}

uint32_t scatter_bins(uint32_t n_tris) {
    // about one bin per triangle; a handful needs no bins
    uint32_t g = 1;
    if (n_tris > 16u)
        while (g < 128u && g * g < n_tris) g += 1u;
    return g;
}

size_t scatter_workspace(uint32_t n_tris) {
    const uint64_t g = scatter_bins(n_tris);
    return 32 + (size_t)n_tris * (3 * 16 + 3 * 16 + 4) + (size_t)(2 * g * g + 1) * 4 + (size_t)scatter_cap(n_tris) * 4;
}

cudaError_t launch_scatter(ScatterArgs a, const float* host_verts, char* ws, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    const size_t nt = a.n_tris;
    a.bins = scatter_bins(a.n_tris);
    a.cap = scatter_cap(a.n_tris);
    const uint32_t nb = a.bins * a.bins;
    // the counters first (one clear), rounded to 16 bytes with what follows
    const size_t head = 16 + ((size_t)nb * 4 + 15) / 16 * 16;
    a.large = reinterpret_cast<unsigned long long*>(ws);
    a.count = reinterpret_cast<uint32_t*>(ws + 16);
    float4* verts = reinterpret_cast<float4*>(ws + head);
    a.verts = verts;
    a.tris = verts + nt * 3;
    a.range = reinterpret_cast<uint32_t*>(a.tris + nt * 3);
    a.start = a.range + nt;
    a.list = a.start + nb + 1;
    for (int k = 0; k < 2; k++) {
        const float ext = a.mmax[k + 1] - a.mmin[k + 1];
        a.blo[k] = a.mmin[k + 1];
        a.binv[k] = ext > 0.f && ext < 3e38f ? (float)a.bins / ext : 0.f;
    }
    cudaError_t e = cudaMemcpyAsync(verts, host_verts, nt * 48, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws, 0, head, s);
    if (e != cudaSuccess) return e;
    const uint32_t tb = (a.n_tris + 3u) / 4u;
    k_sc_prep<<<tb, 128, 0, s>>>(a);
    k_sc_scan<<<1, 1024, 0, s>>>(a);
    k_sc_fill<<<tb, 128, 0, s>>>(a);
    k_scatter<<<(a.n + SCATTER_BS - 1) / SCATTER_BS, SCATTER_BS, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace mpm
