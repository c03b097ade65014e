// mpm_kernels.cu -- the MPM substep as CUDA kernels for sm_100a.
//
// Substep (explicit):  bin_insert -> bin_plan -> bin_scatter
//                      -> p2g_explicit -> g2p_explicit (G2P + integrate fused)
// Substep (PBMPM, n_iter iterations):  same binning, then
//                      pbmpm_first (constraints + affine P2G + forces)
//                      -> (n_iter-1) x pbmpm_iter (G2P, constraints, P2G fused)
//                      -> g2p_pbmpm (last G2P + integrate fused)
//
// The reference runs the same math as 11 (explicit) or 16 (PBMPM, 3 iters)
// WGSL dispatches (src/lib/gpu/mpm/GpuMpmPipelineManager.ts:327-521) with
// 108 global i32 atomics per particle per transfer; here each tile's
// particles accumulate into a shared-memory halo tile and the tile is
// written once with plain 16-byte stores.
#include <algorithm>
#include <type_traits>

#include "mpm_engine.cuh"
#include "mpm_math.cuh"
#include "mpm_plast.cuh"

namespace mpm {

// ------------------------------------------------------------------
// shared helpers
// ------------------------------------------------------------------
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t tile_hash(uint32_t scene, int sx, int sy, int sz) {
    return hash3((uint32_t)sx, (uint32_t)sy, (uint32_t)sz) ^ (scene * 0x9E3779B1u);
}

// Slot of `key`, claimed if the table does not hold it yet; a new slot gets
// the next compact tile index (any order: results do not depend on it), so
// the occupied tiles need no scan of the table.
__device__ uint32_t tile_insert(const Ctx& c, uint64_t key, uint32_t scene, int sx, int sy, int sz) {
    uint32_t mask = c.cap - 1u;
    uint32_t s = tile_hash(scene, sx, sy, sz) & mask;
    uint32_t limit = c.cap < MAX_PROBES ? c.cap : MAX_PROBES;
    for (uint32_t probe = 0; probe < limit; probe++) {
        unsigned long long k = *((volatile unsigned long long*)&c.keys[s]);
        if (k == key) return s;
        if (k == KEY_EMPTY) {
            unsigned long long old = atomicCAS(&c.keys[s], KEY_EMPTY, (unsigned long long)key);
            if (old == KEY_EMPTY) {
                const uint32_t st = atomicAdd(&c.counters->n_ins, 1u);
                c.slot_st[s] = st;
                c.st_slot[st] = s;
                c.st_key[st] = key;
                return s;
            }
            if (old == key) return s;
        }
        s = (s + 1u) & mask;
    }
    atomicOr(&c.counters->status, ST_HASH_FULL);
    return INVALID;
}

__device__ uint32_t tile_lookup(const Ctx& c, uint64_t key, uint32_t scene, int sx, int sy, int sz) {
    uint32_t mask = c.cap - 1u;
    uint32_t s = tile_hash(scene, sx, sy, sz) & mask;
    uint32_t limit = c.cap < MAX_PROBES ? c.cap : MAX_PROBES;
    for (uint32_t probe = 0; probe < limit; probe++) {
        unsigned long long k = c.keys[s];
        if (k == key) return s;
        if (k == KEY_EMPTY) return INVALID;
        s = (s + 1u) & mask;
    }
    return INVALID;
}

__device__ __forceinline__ uint32_t find_scene(const Ctx& c, uint32_t p) {
    uint32_t lo = 0, hi = c.n_scenes;  // answer in [0, n_scenes)
    while (hi - lo > 1u) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&c.scene_first[mid]) <= p) lo = mid; else hi = mid;
    }
    return lo;
}

// floor(a / E) for a compile-time tile edge E (also for negative a)
template <int E>
__device__ __forceinline__ int floor_div(int a) {
    int q = a / E;
    return (a < 0 && q * E != a) ? q - 1 : q;
}

__device__ __forceinline__ void load_scene_smem(SceneDev& dst, const SceneDev* src) {
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
    for (int i = threadIdx.x; i < (int)(sizeof(SceneDev) / 4); i += blockDim.x) d[i] = s[i];
}

// f32(i) / fixedPointScale
__device__ __forceinline__ float inv_s(const SceneDev& S, int32_t v) { return fm(i2f(v), S.rscale); }

// Grid-side boundary of boundary_mode 1 (an extension; the reference only
// reflects particles): sticky ground plane, slip walls.
__device__ __forceinline__ void grid_bc(const SceneDev& S, const int* gc, float* v) {
    if (S.bmode != 1u) return;
    if (gc[S.gaxis] < S.bc) { v[0] = 0.f; v[1] = 0.f; v[2] = 0.f; return; }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (gc[a] < S.bc && v[a] < 0.f) v[a] = 0.f;
        if (gc[a] >= S.res[a] - S.bc && v[a] > 0.f) v[a] = 0.f;
    }
}

// ------------------------------------------------------------------
// particle state access: the record of work slot t, word q at w[q * n + t]
// (mpm_engine.cuh lists the words)
// ------------------------------------------------------------------
struct PState {
    float pos[3], hom, vel[3], mass;
    float Fe[9], Fp[9], dxp[3], D[9];
};

// The particles of one tile for a tile kernel's thread, Q float4 words each, one
// plane per word (SORTED: and the work state's float2): the thread takes the tile's particles threadIdx.x, + BS, ...
// Their slots are read one particle ahead, the first one before the CTA sets
// up the tile, so no particle waits for two dependent loads: set + n substeps +
// get, 32,768 explicit particles 123.7 -> 120.8 us (n = 8), 262,144 PBMPM
// particles 956 -> 937 us (4), 4,194,304 5,410 -> 5,276 us (1).  Copies of the
// next particle's words into shared memory (cp.async) were no faster than that
// (explicit, edge 4: 255 -> 252 us; edge 8 with 512 threads 121 -> 126 us, PBMPM
// 770 -> 823 us): they take the L1's room.
template <int BS, int Q, bool SORTED>
struct Feed {
    const float4* w;          // plane 0
    size_t n;                 // words per plane
    const uint32_t* sorted;   // SORTED: the tile's slots; else the tile's particles are contiguous from w
    uint32_t cnt;
    uint32_t i, pid, nxt;

    __device__ __forceinline__ uint32_t slot(uint32_t k) const { return SORTED ? sorted[k] : k; }
    __device__ __forceinline__ void begin(const float4* planes, size_t words, const uint32_t* order, uint32_t first,
                                          uint32_t count) {
        w = SORTED ? planes : planes + first;
        n = words;
        sorted = SORTED ? order + first : nullptr;
        cnt = count;
        i = threadIdx.x;
        pid = i < cnt ? slot(i) : 0u;
        nxt = i + BS < cnt ? slot(i + BS) : 0u;
    }
    __device__ __forceinline__ bool more() const { return i < cnt; }
    __device__ __forceinline__ void take(float4* r) const {
#pragma unroll
        for (int q = 0; q < Q; q++) r[q] = __ldg(w + q * n + pid);
    }
    __device__ __forceinline__ float2 tail() const { return __ldg(work_tail(w, n) + pid); }
    __device__ __forceinline__ void next() {
        i += BS;
        pid = nxt;
        if (i + BS < cnt) nxt = slot(i + BS);
    }
};

// work words 0..5 and the tail (position, velocity, mass, Fe, Fp) and, of 9,
// words 6..8 (displacement, D)
template <int Q>
__device__ __forceinline__ void unpack_particle(const float4* r, float2 t, PState& s) {
    s.pos[0] = r[0].x; s.pos[1] = r[0].y; s.pos[2] = r[0].z; s.hom = r[0].w;
    s.vel[0] = r[1].x; s.vel[1] = r[1].y; s.vel[2] = r[1].z; s.mass = r[1].w;
    s.Fe[0] = r[2].x; s.Fe[1] = r[2].y; s.Fe[2] = r[2].z; s.Fe[3] = r[2].w;
    s.Fe[4] = r[3].x; s.Fe[5] = r[3].y; s.Fe[6] = r[3].z; s.Fe[7] = r[3].w;
    s.Fe[8] = r[4].x; s.Fp[0] = r[4].y; s.Fp[1] = r[4].z; s.Fp[2] = r[4].w;
    s.Fp[3] = r[5].x; s.Fp[4] = r[5].y; s.Fp[5] = r[5].z; s.Fp[6] = r[5].w;
    s.Fp[7] = t.x; s.Fp[8] = t.y;
    if (Q == 9) {
        s.dxp[0] = r[6].x; s.dxp[1] = r[6].y; s.dxp[2] = r[6].z; s.D[0] = r[6].w;
        s.D[1] = r[7].x; s.D[2] = r[7].y; s.D[3] = r[7].z; s.D[4] = r[7].w;
        s.D[5] = r[8].x; s.D[6] = r[8].y; s.D[7] = r[8].z; s.D[8] = r[8].w;
    }
}

// the words a G2P + integrate writes (the position's fourth word kept), streamed
// past L1
__device__ __forceinline__ void store_particle(float4* w, size_t n, uint32_t t, const PState& s) {
    float4* r = w + t;
    __stcs(r, make_float4(s.pos[0], s.pos[1], s.pos[2], s.hom));
    __stcs(r + n, make_float4(s.vel[0], s.vel[1], s.vel[2], s.mass));
    __stcs(r + 2 * n, make_float4(s.Fe[0], s.Fe[1], s.Fe[2], s.Fe[3]));
    __stcs(r + 3 * n, make_float4(s.Fe[4], s.Fe[5], s.Fe[6], s.Fe[7]));
    __stcs(r + 4 * n, make_float4(s.Fe[8], s.Fp[0], s.Fp[1], s.Fp[2]));
    __stcs(r + 5 * n, make_float4(s.Fp[3], s.Fp[4], s.Fp[5], s.Fp[6]));
    __stcs(r + 6 * n, make_float4(s.dxp[0], s.dxp[1], s.dxp[2], s.D[0]));
    __stcs(r + 7 * n, make_float4(s.D[1], s.D[2], s.D[3], s.D[4]));
    __stcs(r + 8 * n, make_float4(s.D[5], s.D[6], s.D[7], s.D[8]));
    __stcs(work_tail(w, n) + t, make_float2(s.Fp[7], s.Fp[8]));
}

// cell number, fractional position, quadratic B-spline weights
// (mpmOps.wgsl:14-53)
struct Stencil {
    int cell[3];
    float f[3];
    float w[3][3];   // w[k][axis], k = offset + 1
};

__device__ __forceinline__ void make_stencil(const SceneDev& S, const float* pos, Stencil& st) {
#pragma unroll
    for (int i = 0; i < 3; i++) st.cell[i] = f2i(fm(fs(pos[i], S.gmin[i]), S.rcd[i]));
#pragma unroll
    for (int i = 0; i < 3; i++) {
        float mn = ff(S.cd[i], i2f(st.cell[i]), S.gmin[i]);
        float f = fm(fs(pos[i], mn), S.rcd[i]);
        st.f[i] = f;
        float om = fs(1.0f, f);
        st.w[0][i] = fm(fm(0.5f, om), om);
        float h = fs(f, 0.5f);
        st.w[1][i] = ff(-h, h, 0.75f);
        st.w[2][i] = fm(fm(0.5f, f), f);
    }
}

__device__ __forceinline__ float dwk(int k, float f) {
    // derivative of the B-spline weights wrt the fractional position
    return k == 0 ? fs(f, 1.0f) : (k == 1 ? fm(-2.0f, fs(f, 0.5f)) : f);
}

// ------------------------------------------------------------------
// constitutive pieces
// ------------------------------------------------------------------
// hardenLameParameters + calculateStressFirstPiolaKirchhoff
// (stressTensorOps.wgsl:9-22, 39-56); returns M = (-V) * P^T.
__device__ __forceinline__ void stress_matrix(const SceneDev& S, const PState& p, float* M) {
    float Jp = det3(p.Fp);
    float ef = expf_m(fm(S.xi_e, fs(1.0f, Jp)));
    float mu = fm(S.mu0, ef);
    float la = fm(S.la0, ef);
    float J = det3(p.Fe);
    float R[9], Fi[9];
    polar3(p.Fe, R);
    inv3(p.Fe, Fi);
    float a = fm(2.0f, mu);
    float b = fm(fm(la, fs(J, 1.0f)), J);
    float V = fm(p.mass, S.inv_rho);
    float nV = -V;
    // P[c][r] = a*(F[c][r]-R[c][r]) + b*Fi^T[c][r], Fi^T[c][r] = Fi[r][c]
    // M[c][r] = (-V) * P^T[c][r] = (-V) * P[r][c]
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int r = 0; r < 3; r++) {
            float Prc = ff(b, Fi[c * 3 + r], fm(a, fs(p.Fe[r * 3 + c], R[r * 3 + c])));
            M[c * 3 + r] = fm(nV, Prc);
        }
}

// elasticity relaxation factor 0.5 + 0.5 (1 - exp(-xi / det Fp)) (pbmpm.wgsl:29-35)
__device__ __forceinline__ float pbmpm_relax(const SceneDev& S, const float* Fp) {
    float J = det3(Fp);
    return ff(0.5f, fs(1.0f, expf_m(fd(-S.xi_p, J))), 0.5f);
}

// solveParticleConstraints (pbmpm.wgsl:16-39): updates D, given Fe, its
// inverse and the relaxation factor (both fixed within a substep).
__device__ __forceinline__ void pbmpm_constraints(const SceneDev& S, const float* Fe, const float* Fei, float relax,
                                                  float* D) {
    float IpD[9], Ft[9], Rt[9];
#pragma unroll
    for (int i = 0; i < 9; i++) IpD[i] = fa((i == 0 || i == 4 || i == 8) ? 1.0f : 0.0f, D[i]);
    mul3(IpD, Fe, Ft);
    polar3(Ft, Rt);
    float tv = det3(Ft);
    float vs = powf_m(fabsf(tv), S.vexp);
    float ob = fs(1.0f, S.blend);
    float tb[9], Dc[9];
    // tb = blend (R vs) + (1 - blend) R, D += relax (Dc - I - D), in pairs
    const float2 vs2 = dup2(vs), ob2 = dup2(ob), bl2 = dup2(S.blend), rx2 = dup2(relax);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float2 r = make_float2(Rt[i], Rt[i + 1]);
        const float2 v = ff2(bl2, fm2(r, vs2), fm2(ob2, r));
        tb[i] = v.x;
        tb[i + 1] = v.y;
    }
    tb[8] = ff(S.blend, fm(Rt[8], vs), fm(ob, Rt[8]));
    mul3(tb, Fei, Dc);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        const float2 id = make_float2((i == 0 || i == 4) ? 1.0f : 0.0f, (i + 1 == 4) ? 1.0f : 0.0f);
        const float2 d = make_float2(D[i], D[i + 1]);
        const float2 v = ff2(rx2, fa2(fa2(make_float2(Dc[i], Dc[i + 1]), neg2(id)), neg2(d)), d);
        D[i] = v.x;
        D[i + 1] = v.y;
    }
    D[8] = ff(relax, fs(fs(Dc[8], 1.0f), D[8]), D[8]);
}

// applyPlasticity (plasticityOps.wgsl:7-48), in mpm_plast.cuh
__device__ __forceinline__ void plasticity(const SceneDev& S, float* Fe, float* Fp) {
    plasticity_exact(S.smin, S.smax, Fe, Fp);
}

// ------------------------------------------------------------------
// collider (colliderPrelude.wgsl:29-356)
// ------------------------------------------------------------------
__device__ __forceinline__ void col_vertex(const SceneDev& S, uint32_t idx, float* v) {
    uint32_t base = S.c_nidx + idx * 3u;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        uint32_t w = (base + (uint32_t)k < S.col_words) ? __ldg(&S.col_data[base + k]) : 0u;
        v[k] = __uint_as_float(w);
    }
}

__device__ void closest_point_tri(const float* p, const float* a, const float* b, const float* c, float* o) {
    float ab[3], ac[3], ap[3];
#pragma unroll
    for (int k = 0; k < 3; k++) { ab[k] = fs(b[k], a[k]); ac[k] = fs(c[k], a[k]); ap[k] = fs(p[k], a[k]); }
    float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
    if (d1 <= 0.f && d2 <= 0.f) { o[0] = a[0]; o[1] = a[1]; o[2] = a[2]; return; }
    float bp[3];
#pragma unroll
    for (int k = 0; k < 3; k++) bp[k] = fs(p[k], b[k]);
    float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3 >= 0.f && d4 <= d3) { o[0] = b[0]; o[1] = b[1]; o[2] = b[2]; return; }
    float vc = fs(fm(d1, d4), fm(d3, d2));
    if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
        float v = fd(d1, fs(d1, d3));
#pragma unroll
        for (int k = 0; k < 3; k++) o[k] = fa(a[k], fm(v, ab[k]));
        return;
    }
    float cp[3];
#pragma unroll
    for (int k = 0; k < 3; k++) cp[k] = fs(p[k], c[k]);
    float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    if (d6 >= 0.f && d5 <= d6) { o[0] = c[0]; o[1] = c[1]; o[2] = c[2]; return; }
    float vb = fs(fm(d5, d2), fm(d1, d6));
    if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
        float w = fd(d2, fs(d2, d6));
#pragma unroll
        for (int k = 0; k < 3; k++) o[k] = fa(a[k], fm(w, ac[k]));
        return;
    }
    float va = fs(fm(d3, d6), fm(d5, d4));
    if (va <= 0.f && fs(d4, d3) >= 0.f && fs(d5, d6) >= 0.f) {
        float w = fd(fs(d4, d3), fa(fs(d4, d3), fs(d5, d6)));
#pragma unroll
        for (int k = 0; k < 3; k++) o[k] = fa(b[k], fm(w, fs(c[k], b[k])));
        return;
    }
    float denom = fd(1.0f, fa(fa(va, vb), vc));
    float v = fm(vb, denom), w = fm(vc, denom);
#pragma unroll
    for (int k = 0; k < 3; k++) o[k] = fa(fa(a[k], fm(v, ab[k])), fm(w, ac[k]));
}

__device__ float ray_tri(const float* org, const float* dir, const float* a, const float* b, const float* c) {
    const float EPS = 1e-6f;
    float e1[3], e2[3], h[3], sv[3], q[3];
#pragma unroll
    for (int k = 0; k < 3; k++) { e1[k] = fs(b[k], a[k]); e2[k] = fs(c[k], a[k]); }
    cross3(dir, e2, h);
    float aa = dot3(e1, h);
    if (aa > -EPS && aa < EPS) return -1.f;
    float f = fd(1.0f, aa);
#pragma unroll
    for (int k = 0; k < 3; k++) sv[k] = fs(org[k], a[k]);
    float u = fm(f, dot3(sv, h));
    if (u < 0.f || u > 1.f) return -1.f;
    cross3(sv, e1, q);
    float v = fm(f, dot3(dir, q));
    if (v < 0.f || fa(u, v) > 1.f) return -1.f;
    float t = fm(f, dot3(e2, q));
    if (t > EPS) return t;
    return -1.f;
}

// What a collision query reads and changes of a particle.
struct ColState {
    float pos[3], vel[3], dxp[3];
};

// Allowances of the skips below (identity transform only).  A triangle whose
// bounds are farther than the threshold (plus a rounding allowance) from the
// particle and do not meet its path can neither bring the closest distance
// under the threshold nor be hit by the path, so it cannot change the outcome;
// the other triangles run in the same order.
__device__ __forceinline__ float col_slack(const float* cur) {
    return fa(1e-4f, fm(1e-5f, fmaxf(fmaxf(fabsf(cur[0]), fabsf(cur[1])), fabsf(cur[2]))));
}

// False where the query's outcome is "unchanged" without traversing the tree:
// the path misses the collider's box, or (identity transform only) the
// collider's distance field bounds the distance from the particle to every
// triangle from below by more than the threshold plus the path length -- every
// point of the path is then farther than the threshold from every triangle, so
// no triangle can bring the closest distance under it and the path hits none.
__device__ __forceinline__ bool may_collide(const SceneDev& S, const float* cur, const float* dxp) {
    if (S.n_nodes == 0u || S.c_nobj == 0u) return false;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float prev = fs(cur[k], dxp[k]);
        if (fminf(cur[k], prev) > S.cbhi[k] || fmaxf(cur[k], prev) < S.cblo[k]) return false;
    }
    if (S.cull && S.dfield != nullptr) {
        bool in = true;
        uint32_t fc[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float u = fm(fs(cur[k], S.df_lo[k]), S.df_rcs[k]);
            in = in && u >= 0.f && u < (float)S.df_res;
            fc[k] = in ? (uint32_t)u : 0u;
        }
        if (in && fc[0] < S.df_res && fc[1] < S.df_res && fc[2] < S.df_res) {
            const float lb = __ldg(S.dfield + ((size_t)fc[2] * S.df_res + fc[1]) * S.df_res + fc[0]);
            if (lb > fa(fa(S.cthr, col_slack(cur)), len3(dxp))) return false;
        }
    }
    return true;
}

// The query of a particle that may_collide lets through.
__device__ __forceinline__ void collide(const SceneDev& S, ColState& p, Counters* ctr) {
    const float margin = S.cmargin;
    float cur[3], prev[3];
#pragma unroll
    for (int k = 0; k < 3; k++) { cur[k] = p.pos[k]; prev[k] = fs(cur[k], p.dxp[k]); }

    float min_d2 = 1e20f;
    float cnorm[3] = {0.f, 0.f, 1.f}, cpos[3] = {cur[0], cur[1], cur[2]};
    float min_t = 1.f;
    float hnorm[3] = {0.f, 0.f, 1.f}, hpos[3] = {cur[0], cur[1], cur[2]};
    bool has_hit = false;
    float rd[3] = {p.dxp[0], p.dxp[1], p.dxp[2]};
    bool do_ccd = len3(rd) > 1e-4f;
    float curl[3], prevl[3], pminl[3], pmaxl[3];
    xform_point(S.xfi, cur, curl);
    xform_point(S.xfi, prev, prevl);
#pragma unroll
    for (int k = 0; k < 3; k++) { pminl[k] = fminf(curl[k], prevl[k]); pmaxl[k] = fmaxf(curl[k], prevl[k]); }

    const float slack = col_slack(cur);
    const float reach = fa(S.cthr, slack);
    const float reach2 = fm(reach, reach);
    // with the triangle records: a triangle farther than the closest distance
    // so far plus the allowance cannot become the closest either (near2);
    // bn: the last closest triangle with a normal
    float near2 = reach2;
    uint32_t bn = INVALID;
    float seg_lo[3], seg_hi[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        seg_lo[k] = fs(fminf(cur[k], prev[k]), slack);
        seg_hi[k] = fa(fmaxf(cur[k], prev[k]), slack);
    }
    uint32_t stack[32];
    uint32_t sp = 0;
    stack[sp++] = 0u;
    // a well-formed tree visits each node at most once; the cap only ends
    // traversal of a malformed (cyclic) node array
    uint32_t visits = 0, max_visits = 2u * S.n_nodes + 64u;
    while (sp > 0u) {
        if (++visits > max_visits) { atomicOr(&ctr->status, ST_BVH_STACK); break; }
        uint32_t ni = stack[--sp];
        if (ni >= S.n_nodes) continue;
        const uint4* nd = reinterpret_cast<const uint4*>(S.bvh + (size_t)ni * 8);
        uint4 n0 = __ldg(nd), n1 = __ldg(nd + 1);
        float bmin0 = fs(__uint_as_float(n0.x), margin), bmin1 = fs(__uint_as_float(n0.y), margin), bmin2 = fs(__uint_as_float(n0.z), margin);
        float bmax0 = fa(__uint_as_float(n1.x), margin), bmax1 = fa(__uint_as_float(n1.y), margin), bmax2 = fa(__uint_as_float(n1.z), margin);
        if (pminl[0] > bmax0 || pminl[1] > bmax1 || pminl[2] > bmax2 ||
            pmaxl[0] < bmin0 || pmaxl[1] < bmin1 || pmaxl[2] < bmin2) continue;
        if (n1.w & 0x80000000u) {
            uint32_t start = n0.w, end = start + (n1.w & 0x7FFFFFFFu);
            for (uint32_t i = start; i < end; i++) {
                uint32_t tb = i * 3u;
                if (tb + 2u >= S.col_words) break;
                const float4* rec = S.tbox + (size_t)TRI_WORDS * i;
                float v0[3], v1[3], v2[3];
                bool has_normal = false;
                if (S.cull) {
                    const float4 blo = __ldg(rec), bhi = __ldg(rec + 1);
                    const float lo3[3] = {blo.x, blo.y, blo.z}, hi3[3] = {bhi.x, bhi.y, bhi.z};
                    float dl = 0.f;
                    bool apart = false;
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        float gap = fmaxf(0.f, fmaxf(fs(lo3[k], cur[k]), fs(cur[k], hi3[k])));
                        dl = fa(dl, fm(gap, gap));
                        apart = apart || seg_hi[k] < lo3[k] || seg_lo[k] > hi3[k];
                    }
                    // The closest point's barycentrics are off by about
                    // 16 ulp * L^2 (L + distance)^2 / |n|^2 (L: longest edge,
                    // n: edge cross product), the point by L times that;
                    // below half the allowance (bhi.w = L^3 / |n|^2) the
                    // computed distance cannot undercut the bounds'.
                    const float lr = fa(blo.w, reach);
                    const float lim2 = fm(bhi.w, fm(lr, lr)) < 50.0f ? near2 : reach2;
                    if (dl > lim2 && (!do_ccd || apart)) continue;
                    const float4 a = __ldg(rec + 2), b = __ldg(rec + 3), d = __ldg(rec + 4);
                    v0[0] = a.x; v0[1] = a.y; v0[2] = a.z;
                    v1[0] = b.x; v1[1] = b.y; v1[2] = b.z;
                    v2[0] = d.x; v2[1] = d.y; v2[2] = d.z;
                    has_normal = a.w != 0.f;
                } else {
                    float v0l[3], v1l[3], v2l[3];
                    col_vertex(S, __ldg(&S.col_data[tb]), v0l);
                    col_vertex(S, __ldg(&S.col_data[tb + 1]), v1l);
                    col_vertex(S, __ldg(&S.col_data[tb + 2]), v2l);
                    xform_point(S.xf, v0l, v0);
                    xform_point(S.xf, v1l, v1);
                    xform_point(S.xf, v2l, v2);
                }
                float cp[3], df[3];
                closest_point_tri(cur, v0, v1, v2, cp);
#pragma unroll
                for (int k = 0; k < 3; k++) df[k] = fs(cur[k], cp[k]);
                float d2 = dot3(df, df);
                if (d2 < min_d2) {
                    min_d2 = d2;
                    cpos[0] = cp[0]; cpos[1] = cp[1]; cpos[2] = cp[2];
                    if (S.cull) {
                        const float nr = fa(__fsqrt_rn(d2), slack);
                        near2 = fminf(reach2, fm(nr, nr));
                        if (has_normal) bn = i;
                    } else {
                        float n[3];
                        const float ln = tri_normal(v0, v1, v2, n);
                        if (ln > 1e-6f) {
#pragma unroll
                            for (int k = 0; k < 3; k++) cnorm[k] = fd(n[k], ln);
                        }
                    }
                }
                if (do_ccd) {
                    float t = ray_tri(prev, rd, v0, v1, v2);
                    if (t > 0.f && t < min_t) {
                        min_t = t;
                        has_hit = true;
#pragma unroll
                        for (int k = 0; k < 3; k++) hpos[k] = fa(prev[k], fm(rd[k], t));
                        float n[3];
                        const float ln = tri_normal(v0, v1, v2, n);
                        float fn[3] = {fd(n[0], ln), fd(n[1], ln), fd(n[2], ln)};
                        float dd = dot3(rd, fn);
                        float sg = dd > 0.f ? 1.f : (dd < 0.f ? -1.f : 0.f);
#pragma unroll
                        for (int k = 0; k < 3; k++) hnorm[k] = fm(fn[k], sg);
                    }
                }
            }
        } else {
            if (sp < 31u) {
                stack[sp++] = n0.w;
                stack[sp++] = n1.w;
            } else {
                atomicOr(&ctr->status, ST_BVH_STACK);
            }
        }
    }
    float vsf = fm(S.cvs, S.rdt);
    if (has_hit) {
        float nvv[3], vr[3];
#pragma unroll
        for (int k = 0; k < 3; k++) p.pos[k] = fa(hpos[k], fm(hnorm[k], S.csurf));
#pragma unroll
        for (int k = 0; k < 3; k++) vr[k] = fs(fm(p.dxp[k], S.rdt), S.cvel[k]);
        float vn = dot3(vr, hnorm);
        float om = fs(1.0f, S.cfric);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float vt = fs(vr[k], fm(vn, hnorm[k]));
            nvv[k] = vn < 0.f ? fa(fm(vt, om), fm(S.cvel[k], vsf)) : fa(vr[k], fm(S.cvel[k], vsf));
        }
#pragma unroll
        for (int k = 0; k < 3; k++) { p.vel[k] = nvv[k]; p.dxp[k] = fm(nvv[k], S.dt); }
        return;
    }
    float dist = __fsqrt_rn(min_d2);
    if (!(dist < S.cthr)) return;
    if (bn != INVALID) {
        const float4 nn = __ldg(S.tbox + (size_t)TRI_WORDS * bn + 5);
        cnorm[0] = nn.x; cnorm[1] = nn.y; cnorm[2] = nn.z;
    }
    float df[3], pd[3] = {cnorm[0], cnorm[1], cnorm[2]};
#pragma unroll
    for (int k = 0; k < 3; k++) df[k] = fs(cur[k], cpos[k]);
    float ld = len3(df);
    if (ld > 1e-6f) {
#pragma unroll
        for (int k = 0; k < 3; k++) pd[k] = fd(df[k], ld);
    }
    if (dist < S.cthr) {
        float nvv[3], vr[3];
#pragma unroll
        for (int k = 0; k < 3; k++) vr[k] = fs(fm(p.dxp[k], S.rdt), S.cvel[k]);
        float vn = dot3(vr, pd);
        float om = fs(1.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float vt = fs(vr[k], fm(vn, pd[k]));
            nvv[k] = vn < 0.f ? fa(fm(vt, om), fm(S.cvel[k], vsf)) : fa(vr[k], fm(S.cvel[k], vsf));
        }
#pragma unroll
        for (int k = 0; k < 3; k++) { p.vel[k] = nvv[k]; p.dxp[k] = fm(nvv[k], S.dt); }
        if (dist < S.csurf) {
#pragma unroll
            for (int k = 0; k < 3; k++) p.pos[k] = fa(cpos[k], fm(pd[k], S.csurf));
        }
    }
}

// Appends work_out slot pid to a list of the passes after the G2P
// (warp-aggregated).
__device__ __forceinline__ void append(uint32_t* list, uint32_t* n, uint32_t pid) {
    unsigned m = __activemask();
    int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(n, (uint32_t)__popc(m));
    base = __shfl_sync(m, base, leader);
    list[base + (uint32_t)__popc(m & lanemask_lt())] = pid;
}

// integrateParticles (integrateParticles.wgsl:14-72).  The return map runs
// only for particles the strain-bound check does not clear (for the others it
// returns Fe and Fp unchanged, bit for bit).  With deferred plasticity the
// record keeps the trial Fe and those particles are listed for the plasticity
// pass (exact or learned).  Particles that the collider may touch are listed
// for the collision pass (k_collide).
__device__ __forceinline__ void integrate(const Ctx& c, const SceneDev& S, PState& p, uint32_t pid) {
#pragma unroll
    for (int k = 0; k < 3; k++) p.pos[k] = fa(p.pos[k], p.dxp[k]);
    float IpD[9];
#pragma unroll
    for (int i = 0; i < 9; i++) IpD[i] = fa((i == 0 || i == 4 || i == 8) ? 1.0f : 0.0f, p.D[i]);
    mul3(IpD, p.Fe, p.Fe);
    const bool certified = cert_elastic(S.smin, S.smax, p.Fe);
    if (c.plast_defer) {
        if (!certified) append(c.plast_list, &c.counters->n_plast, pid);
    } else if (!certified) {
        plasticity(S, p.Fe, p.Fp);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (p.pos[a] < S.gmin[a]) { p.dxp[a] = fm(p.dxp[a], S.rest); p.pos[a] = S.gmin[a]; p.vel[a] = fm(p.vel[a], S.rest); }
        if (p.pos[a] >= S.gmax[a]) { p.dxp[a] = fm(p.dxp[a], S.rest); p.pos[a] = S.gmax[a]; p.vel[a] = fm(p.vel[a], S.rest); }
    }
    if (may_collide(S, p.pos, p.dxp)) append(c.col_list, &c.counters->n_col, pid);
}

// The collision query (colliderPrelude.wgsl:29-356) of the particles the G2P
// listed, one thread each.  Bound by the latency of the tree traversal and by
// lanes of a warp that traverse different depths.  Its own pass because the
// particles near a collider sit in a few tiles: inside the G2P they held up
// those tiles' CTAs while the other SMs ran out of work (SMs active for 29 %
// of the launch on a 524,288-particle slab lying on a 130,050-triangle
// terrain), and the traversal's registers limited every tile CTA's occupancy.
// Consecutive list entries come from one tile, so a warp's paths lie close
// together.
__global__ void __launch_bounds__(128) k_collide(Ctx c) {
    __shared__ SceneDev S1;
    const uint32_t n_list = c.counters->n_col;
    if (blockIdx.x * 128u >= n_list) return;
    if (c.n_scenes == 1u) load_scene_smem(S1, c.scenes);
    __syncthreads();
    const size_t n = c.n_particles;
    for (uint32_t i = blockIdx.x * 128u + threadIdx.x; i < n_list; i += gridDim.x * 128u) {
        const uint32_t t = c.col_list[i];
        const SceneDev& S = c.n_scenes == 1u ? S1 : c.scenes[find_scene(c, c.ids_out[t])];
        float4* r = c.work_out + t;
        const float4 q0 = r[0], q1 = r[n], q6 = r[6 * n];
        ColState p = {{q0.x, q0.y, q0.z}, {q1.x, q1.y, q1.z}, {q6.x, q6.y, q6.z}};
        collide(S, p, c.counters);
        r[0] = make_float4(p.pos[0], p.pos[1], p.pos[2], q0.w);
        r[n] = make_float4(p.vel[0], p.vel[1], p.vel[2], q1.w);
        r[6 * n] = make_float4(p.dxp[0], p.dxp[1], p.dxp[2], q6.w);
    }
}

// ------------------------------------------------------------------
// binning kernels
// ------------------------------------------------------------------
// Empties the tile table after a binning pass that no bin_scatter follows (the
// sizing passes).
__global__ void k_clear_table(Ctx c) {
    const uint32_t n = c.counters->n_st;
    if (blockIdx.x == 0 && threadIdx.x == 0) c.counters->n_ins = 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t s = c.st_slot[i];
        c.keys[s] = KEY_EMPTY;
        c.slot_count[s] = 0u;
    }
}

template <int E>
__global__ void __launch_bounds__(256) k_bin_insert(Ctx c) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    bool act = t < c.n_particles;
    uint64_t key = KEY_EMPTY;
    uint32_t scene = 0;
    int st[3] = {0, 0, 0};
    if (act) {
        float4 q0 = __ldg(c.work_in + t);
        scene = c.n_scenes > 1u ? find_scene(c, __ldg(c.ids_in + t) & ~ID_KEEP) : 0u;
        const SceneDev* S = c.scenes + scene;
        float pos[3] = {q0.x, q0.y, q0.z};
#pragma unroll
        for (int i = 0; i < 3; i++) {
            int cell = f2i(fm(fs(pos[i], __ldg(&S->gmin[i])), __ldg(&S->rcd[i])));
            int res = __ldg(&S->res[i]);
            // cells below -1 or above res reach no grid cell; clamping them
            // only decides which tile processes the particle
            cell = max(-2, min(cell, res + 1));
            st[i] = floor_div<E>(cell);
        }
        key = pack_key(scene, st[0], st[1], st[2]);
    }
    unsigned am = __ballot_sync(0xffffffffu, act);
    if (!act) return;
    unsigned grp = __match_any_sync(am, key);
    int leader = __ffs(grp) - 1;
    int lane = threadIdx.x & 31;
    uint32_t slot = 0, base = 0;
    if (lane == leader) {
        slot = tile_insert(c, key, scene, st[0], st[1], st[2]);
        base = (slot != INVALID) ? atomicAdd(&c.slot_count[slot], (uint32_t)__popc(grp)) : 0u;
    }
    slot = __shfl_sync(grp, slot, leader);
    base = __shfl_sync(grp, base, leader);
    c.bin_slot[t] = slot;
    c.bin_rank[t] = base + (uint32_t)__popc(grp & lanemask_lt());
}

// Places work slot t at its position in this substep's tile order.  A
// particle that no tile kernel will advance (no hash slot, or a tile past the
// tile storage: both reported in the status) is copied unchanged to its
// output slot, so the state stays complete.  Also empties the tile table
// again (its last reader, bin_plan, is done; there are at most as many tiles
// as particles), so a substep needs no clearing pass of its own.
__global__ void __launch_bounds__(256) k_bin_scatter(Ctx c) {
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c.n_particles) return;
    const uint32_t n_st = c.counters->n_st;
    uint32_t slot = c.bin_slot[t];
    uint32_t dst;
    bool carry = false;
    if (t < n_st) {
        const uint32_t s = c.st_slot[t];
        c.keys[s] = KEY_EMPTY;
        c.slot_count[s] = 0u;
        if (t == 0) c.counters->n_ins = 0u;
    }
    if (slot == INVALID) {
        dst = c.counters->n_binned + atomicAdd(&c.counters->n_carry, 1u);
        carry = true;
    } else {
        dst = c.slot_off[slot] + c.bin_rank[t];
        c.sorted[dst] = t;
        if (n_st > c.max_tiles) carry = c.slot_st[slot] >= c.max_tiles;
    }
    if (carry) {
        const size_t n = c.n_particles;
#pragma unroll
        for (int q = 0; q < WORK_PLANES; q++) c.work_out[q * n + dst] = c.work_in[q * n + t];
        work_tail(c.work_out, n)[dst] = work_tail(c.work_in, n)[t];
        c.ids_out[dst] = c.ids_in[t];
    }
}

// ------------------------------------------------------------------
// tile helpers
// ------------------------------------------------------------------
template <int E>
struct TileCtx {
    uint32_t scene;
    int origin[3];  // first core cell
    uint64_t key;
};

template <int E>
__device__ __forceinline__ void tile_begin(const Ctx& c, uint32_t st, SceneDev& S, TileCtx<E>& T, uint32_t& cur_scene) {
    uint64_t key = c.st_key[st];
    uint32_t scene;
    int sx, sy, sz;
    unpack_key(key, scene, sx, sy, sz);
    T.scene = scene;
    T.key = key;
    T.origin[0] = sx * E; T.origin[1] = sy * E; T.origin[2] = sz * E;
    if (scene != cur_scene) {
        __syncthreads();
        load_scene_smem(S, c.scenes + scene);
        cur_scene = scene;
    }
}

__device__ __forceinline__ int4 add4(int4 s, int4 v) {
    s.x = (int)((uint32_t)s.x + (uint32_t)v.x);
    s.y = (int)((uint32_t)s.y + (uint32_t)v.y);
    s.z = (int)((uint32_t)s.z + (uint32_t)v.z);
    s.w = (int)((uint32_t)s.w + (uint32_t)v.w);
    return s;
}

// Sum of all tile halos covering cell j of this tile's (E+2)^3 region, read
// cell by cell from global memory (inspection kernel only).
template <int E>
__device__ __forceinline__ int4 assemble_cell(const int4* tiles, const int* nbr, int j) {
    constexpr int H = E + 2, NC = H * H * H;
    int lx = j % H, ly = (j / H) % H, lz = j / (H * H);
    int4 s = __ldg(&tiles[(size_t)nbr[13] * NC + j]);
    int dx0 = lx <= 1 ? -1 : 0, dx1 = lx >= E ? 1 : 0;
    int dy0 = ly <= 1 ? -1 : 0, dy1 = ly >= E ? 1 : 0;
    int dz0 = lz <= 1 ? -1 : 0, dz1 = lz >= E ? 1 : 0;
    for (int dz = dz0; dz <= dz1; dz++)
        for (int dy = dy0; dy <= dy1; dy++)
            for (int dx = dx0; dx <= dx1; dx++) {
                if (dx == 0 && dy == 0 && dz == 0) continue;
                int t = nbr[(dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)];
                if (t < 0) continue;
                int jj = ((lz - E * dz) * H + (ly - E * dy)) * H + (lx - E * dx);
                s = add4(s, __ldg(&tiles[(size_t)t * NC + jj]));
            }
    return s;
}

// Compact indices of this tile's 27 neighbours (built by k_tile_nbr) into
// shared memory; d = 9(dz+1) + 3(dy+1) + (dx+1), -1 where no tile exists.
__device__ __forceinline__ void load_neighbors(const Ctx& c, uint32_t st, int* nbr) {
    if (threadIdx.x < 27) nbr[threadIdx.x] = __ldg(&c.st_nbr[(size_t)st * 27u + threadIdx.x]);
}

// Cell velocity the G2P kernels read.  Explicit mode first applies the grid
// update (gridUpdate.cs.wgsl:15-53) with its i32 round trip; PBMPM reads the
// transferred momentum directly (gridToParticle.cs.wgsl:102-108).  Cells the
// reference skips (outside the grid, or mass <= 0) get velocity 0.
// INNER: the cell is inside the grid and out of the boundary's reach.
template <bool PB, bool INNER>
__device__ __forceinline__ float4 cell_velocity(const SceneDev& S, int4 s, const int* gc) {
    const bool in = INNER || (gc[0] >= 0 && gc[1] >= 0 && gc[2] >= 0 && gc[0] < S.res[0] && gc[1] < S.res[1] && gc[2] < S.res[2]);
    float cm = inv_s(S, s.x);
    if (!in || cm <= 0.0f) return make_float4(0.f, 0.f, 0.f, 0.f);
    float rm = __frcp_rn(cm);
    int32_t mi[3] = {s.y, s.z, s.w};
    if (!PB) {
        float u[3];
#pragma unroll
        for (int k = 0; k < 3; k++) u[k] = fa(fm(inv_s(S, mi[k]), rm), S.gdt[k]);
        if (!INNER) grid_bc(S, gc, u);
#pragma unroll
        for (int k = 0; k < 3; k++) mi[k] = f2i(fm(fm(u[k], cm), S.scale));
    }
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; k++) v[k] = fm(inv_s(S, mi[k]), rm);
    if (PB && !INNER) grid_bc(S, gc, v);
    return make_float4(v[0], v[1], v[2], 0.f);
}

// The parts of the 26 neighbour tiles' halos that overlap this tile's
// (E+2)^3 region, flattened into one index space: 6 face slabs (2 x H x H),
// then 12 edge bars (2 x 2 x H), then 8 corner cubes (2 x 2 x 2).  Entry e
// maps to the neighbour direction d (0..26), the cell j of this region and
// the cell jj of the neighbour's region; every divisor is a compile-time
// constant.
template <int E>
struct HaloEntries {
    static constexpr int H = E + 2;
    static constexpr int FACE = 2 * H * H, EDGE = 4 * H;
    static constexpr int NF = 6 * FACE, NED = 12 * EDGE;
    static constexpr int N = NF + NED + 64;
};

template <int E>
__host__ __device__ constexpr void halo_entry(int e, int& d, int& j, int& jj) {
    constexpr int H = E + 2;
    using HE = HaloEntries<E>;
    int dx = 0, dy = 0, dz = 0, ix = 0, iy = 0, iz = 0;
    if (e < HE::NF) {
        int r = e / HE::FACE, o = e - r * HE::FACE;
        int axis = r >> 1, sg = (r & 1) ? 1 : -1;
        if (axis == 0) { ix = o & 1; iy = (o >> 1) % H; iz = (o >> 1) / H; dx = sg; }
        else if (axis == 1) { ix = o % H; iy = (o / H) & 1; iz = o / (2 * H); dy = sg; }
        else { ix = o % H; iy = (o / H) % H; iz = o / (H * H); dz = sg; }
    } else if (e < HE::NF + HE::NED) {
        int e2 = e - HE::NF;
        int r = e2 / HE::EDGE, o = e2 - r * HE::EDGE;
        int za = r >> 2, s1 = (r & 1) ? 1 : -1, s2 = (r & 2) ? 1 : -1;
        if (za == 0) { ix = o % H; iy = (o / H) & 1; iz = o / (2 * H); dy = s1; dz = s2; }
        else if (za == 1) { ix = o & 1; iy = (o >> 1) % H; iz = (o >> 1) / H; dx = s1; dz = s2; }
        else { ix = o & 1; iy = (o >> 1) & 1; iz = o >> 2; dx = s1; dy = s2; }
    } else {
        int o = e - HE::NF - HE::NED;
        int r = o >> 3;
        o &= 7;
        dx = (r & 1) ? 1 : -1; dy = (r & 2) ? 1 : -1; dz = (r & 4) ? 1 : -1;
        ix = o & 1; iy = (o >> 1) & 1; iz = o >> 2;
    }
    int lx = (dx > 0 ? E : 0) + ix, ly = (dy > 0 ? E : 0) + iy, lz = (dz > 0 ? E : 0) + iz;
    j = (lz * H + ly) * H + lx;
    jj = ((lz - E * dz) * H + (ly - E * dy)) * H + (lx - E * dx);
    d = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
}

// The halo entries decoded once, at compile time: entry e packs its
// neighbour direction d (5 bits), its cell j in this tile's region (13 bits)
// and the cell jj in the neighbour's region (13 bits).
template <int E>
struct HaloTable {
    uint32_t v[HaloEntries<E>::N];
};
static_assert((18 * 18 * 18) < (1 << 13), "halo cell index must fit 13 bits");

template <int E>
__host__ __device__ constexpr HaloTable<E> make_halo_table() {
    HaloTable<E> t{};
    for (int e = 0; e < HaloEntries<E>::N; e++) {
        int d = 0, j = 0, jj = 0;
        halo_entry<E>(e, d, j, jj);
        t.v[e] = (uint32_t)d | ((uint32_t)j << 5) | ((uint32_t)jj << 18);
    }
    return t;
}

__device__ const HaloTable<4> g_halo4 = make_halo_table<4>();
__device__ const HaloTable<8> g_halo8 = make_halo_table<8>();
__device__ const HaloTable<12> g_halo12 = make_halo_table<12>();
__device__ const HaloTable<14> g_halo14 = make_halo_table<14>();
__device__ const HaloTable<16> g_halo16 = make_halo_table<16>();

template <int E>
__device__ __forceinline__ const uint32_t* halo_table() {
    return E == 4 ? g_halo4.v : E == 8 ? g_halo8.v : (E == 12 ? g_halo12.v : (E == 14 ? g_halo14.v : g_halo16.v));
}

// ---- TMA bulk copies into shared memory, completing on an mbarrier ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init1(uint64_t* mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes) : "memory");
}
// global -> shared, `bytes` a multiple of 16, both addresses 16-byte aligned
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(mbar))
                 : "memory");
}
// waits for the phase of the given parity; false after `limit` polls
__device__ __forceinline__ bool mbar_wait_parity(uint64_t* mbar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}\n"
            : "=r"(done)
            : "r"(smem_u32(mbar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
constexpr uint32_t COPY_WAIT_LIMIT = 1u << 22;

// Per-CTA state of the halo copies of the tile kernels: the mbarrier the
// bulk copies complete on and the parity of its current phase.
struct HaloCopy {
    uint64_t* mbar;
    uint32_t parity;
};

// Thread 0 issues the bulk copies of tile st's own (E+2)^3 sums into shared
// memory; they complete on hc's mbarrier.
template <int E>
__device__ __forceinline__ void halo_issue(const int4* tiles, uint32_t st, int4* cell, HaloCopy& hc) {
    constexpr int H = E + 2, NC = H * H * H;
    if (threadIdx.x == 0) {
        const int4* own = tiles + (size_t)st * NC;
        // the previous tile's shared-memory reads (generic proxy) come before these writes
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(hc.mbar, (uint32_t)(NC * 16));
        constexpr uint32_t CH = (NC * 16) / 4 / 16 * 16;   // four chunks, 16-byte multiples
        bulk_g2s(cell, own, CH, hc.mbar);
        bulk_g2s(reinterpret_cast<char*>(cell) + CH, reinterpret_cast<const char*>(own) + CH, CH, hc.mbar);
        bulk_g2s(reinterpret_cast<char*>(cell) + 2 * CH, reinterpret_cast<const char*>(own) + 2 * CH, CH, hc.mbar);
        bulk_g2s(reinterpret_cast<char*>(cell) + 3 * CH, reinterpret_cast<const char*>(own) + 3 * CH,
                 (uint32_t)(NC * 16) - 3 * CH, hc.mbar);
    }
}

// Sum this tile's halo region into `cell`: the tile's own (E+2)^3 sums (one
// TMA bulk copy) plus the overlapping parts of the neighbour halos (entries
// of the compile-time halo table, loaded into registers in batches of U per
// thread and added with shared i32 atomics).  The first batch of neighbour
// loads is issued before the wait for the bulk copy, so both latencies
// overlap.  MASS = false adds only the momentum components: the mass field
// of the result keeps the tile's own record (in the PBMPM iterations' halo
// records, the reciprocal cell mass).  Returns false (on every thread) when
// the copy wait ran out; the caller then stops.  PRE = true: the caller issued
// the own-halo copies earlier (halo_issue).
template <int E, int BS, bool MASS = true, bool PRE = false>
__device__ __forceinline__ bool assemble_sums(const int4* tiles, const int* nbr, int4* cell, HaloCopy& hc) {
    constexpr int H = E + 2, NC = H * H * H;
    constexpr int NE = HaloEntries<E>::N;
    constexpr int PER = (NE + BS - 1) / BS;      // entries per thread
    constexpr int U = PER <= 10 ? PER : 8;       // entries per register batch
    const uint32_t* tab = halo_table<E>();
    if (!PRE) halo_issue<E>(tiles, (uint32_t)nbr[13], cell, hc);
    int4 v[U];
    int jd[U];
    auto fetch = [&](int base) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            int e = base + u * BS;
            jd[u] = -1;
            v[u] = make_int4(0, 0, 0, 0);
            if (e < NE) {
                uint32_t w = __ldg(tab + e);
                int t = nbr[w & 31u];
                if (t >= 0) {
                    v[u] = __ldg(tiles + (size_t)t * NC + (w >> 18));
                    jd[u] = (int)((w >> 5) & 0x1fffu);
                }
            }
        }
    };
    auto add = [&]() {
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (jd[u] >= 0) {
                int* dst = reinterpret_cast<int*>(&cell[jd[u]]);
                if (MASS) atomicAdd(dst + 0, v[u].x);
                atomicAdd(dst + 1, v[u].y);
                atomicAdd(dst + 2, v[u].z);
                atomicAdd(dst + 3, v[u].w);
            }
        }
    };
    fetch(threadIdx.x);
    bool ok = mbar_wait_parity(hc.mbar, hc.parity, COPY_WAIT_LIMIT);
    hc.parity ^= 1u;
    if (__syncthreads_or(ok ? 0 : 1)) return false;
    add();
    for (int base = threadIdx.x + U * BS; base < NE; base += U * BS) {
        fetch(base);
        add();
    }
    return true;
}

// Reciprocal cell mass RN(1 / m) of the velocity m^-1 p, 0 for the cells the
// reference skips (outside the grid or mass <= 0): a momentum scaled by 0
// gives a velocity of +-0, whose products add nothing to the G2P sums.
template <bool INNER>
__device__ __forceinline__ float mass_recip(const SceneDev& S, int32_t m, const int* gc) {
    const bool in = INNER || (gc[0] >= 0 && gc[1] >= 0 && gc[2] >= 0 && gc[0] < S.res[0] && gc[1] < S.res[1] && gc[2] < S.res[2]);
    float cm = inv_s(S, m);
    return (in && cm > 0.0f) ? __frcp_rn(cm) : 0.0f;
}

// PBMPM cell velocity from momentum and the reciprocal mass (gridToParticle.cs.wgsl:102-108)
template <bool INNER>
__device__ __forceinline__ float4 cell_velocity_rm(const SceneDev& S, int4 s, float rm, const int* gc) {
    float v[3] = {fm(inv_s(S, s.y), rm), fm(inv_s(S, s.z), rm), fm(inv_s(S, s.w), rm)};
    if (!INNER) grid_bc(S, gc, v);
    return make_float4(v[0], v[1], v[2], 0.f);
}

// Whether a tile's whole halo region lies inside the grid and out of the grid
// boundary's reach, so that its cells need neither coordinates nor checks: the
// conversion of the halo sums took a seventh of a sparse iteration's
// instructions, and most tiles of most scenes are of this kind.  Set + n
// substeps + get: 4,194,304 PBMPM particles 4,880 -> 4,668 us (n = 1), 524,288
// 717 -> 659 (1), 262,144 dense ones 916 -> 904 (4); 1,000,003 explicit 644 ->
// 631 (4), 48 scenes 550 -> 536 us (4).
template <int E>
__device__ __forceinline__ bool inner_tile(const SceneDev& S, const TileCtx<E>& T) {
    const int b = S.bmode == 1u ? max(S.bc, 0) : 0;
    bool inner = true;
#pragma unroll
    for (int k = 0; k < 3; k++) inner = inner && T.origin[k] - 1 >= b && T.origin[k] + E < S.res[k] - b;
    return inner;
}

// Assemble this tile's (E+2)^3 cell velocities in shared memory: halo sums
// (assemble_sums), then each sum turned into the velocity in place.  RM
// selects where the cell masses come from: 0, the assembled mass sums (the
// reference path, explicit grid update included); 1, the same, and the
// reciprocal masses RN(1/m) are kept in rm_s for the tile's flush; 2, the
// reciprocal masses carried in the mass word of the tile's own halo record
// (written there by the previous PBMPM iteration's flush; the halo sums then
// carry momentum only), also kept in rm_s when it is given.  Returns false (on
// every thread) when the halo copy wait ran out.
template <int E, int BS, bool PB, int RM = 0, bool PRE = false>
__device__ __forceinline__ bool assemble_velocity_tile(const int4* tiles, const SceneDev& S, const TileCtx<E>& T,
                                                       const int* nbr, int4* cell, HaloCopy& hc,
                                                       float* rm_s = nullptr) {
    constexpr int H = E + 2, NC = H * H * H;
    if (!assemble_sums<E, BS, RM != 2, PRE>(tiles, nbr, cell, hc)) return false;
    __syncthreads();
    // batches of CB cells per thread: all loads, then all conversions, then
    // all stores, so the cells' dependency chains overlap
    constexpr int CB = (BS >= 512 && RM != 0) ? 4 : 1;
    auto convert = [&](auto inner) {
        constexpr bool INNER = decltype(inner)::value;
        for (int j0 = threadIdx.x; j0 < NC; j0 += CB * BS) {
            int4 sm[CB];
            float rmu[CB];
#pragma unroll
            for (int u = 0; u < CB; u++) {
                int j = j0 + u * BS;
                sm[u] = j < NC ? cell[j] : make_int4(0, 0, 0, 0);
                rmu[u] = (RM == 2 && j < NC) ? __int_as_float(sm[u].x) : 0.0f;
            }
            float4 v[CB];
#pragma unroll
            for (int u = 0; u < CB; u++) {
                int j = j0 + u * BS;
                int gc[3] = {0, 0, 0};
                if (!INNER) {
                    gc[0] = T.origin[0] - 1 + j % H;
                    gc[1] = T.origin[1] - 1 + (j / H) % H;
                    gc[2] = T.origin[2] - 1 + j / (H * H);
                }
                if (RM == 0) {
                    v[u] = cell_velocity<PB, INNER>(S, sm[u], gc);
                } else {
                    float rm;
                    if (RM == 1) {
                        rm = mass_recip<INNER>(S, sm[u].x, gc);
                    } else {
                        rm = rmu[u];
                    }
                    if (rm_s != nullptr && j < NC) rm_s[j] = rm;
                    v[u] = cell_velocity_rm<INNER>(S, sm[u], rm, gc);
                }
            }
#pragma unroll
            for (int u = 0; u < CB; u++) {
                int j = j0 + u * BS;
                if (j < NC) reinterpret_cast<float4*>(cell)[j] = v[u];
            }
        }
    };
    if (inner_tile<E>(S, T)) convert(std::true_type{});
    else convert(std::false_type{});
    return true;
}

// G2P gather from the shared velocity tile (gridToParticle.cs.wgsl:28-130).
// Cells the reference skips hold velocity 0 here: each of their terms is a
// product with a zero factor, and adding +-0 to a sum that started at +0
// leaves it unchanged, so the sums are equal.  The summation order is the
// reference's loop order (z outermost, x innermost).
template <int E, bool PB>
__device__ __forceinline__ void g2p_gather(const TileCtx<E>& T, const float4* vel, const Stencil& sc, float* nv,
                                           float* G) {
    constexpr int H = E + 2;
#pragma unroll
    for (int k = 0; k < 3; k++) nv[k] = 0.f;
#pragma unroll
    for (int i = 0; i < 9; i++) G[i] = 0.f;
    int l0[3];
    bool inside = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        l0[k] = sc.cell[k] - T.origin[k];
        inside = inside && l0[k] >= 0 && l0[k] < E;
    }
    if (!inside) return;
    float offs[3][3];  // offs[axis][o] = (cell + o - 1) - particle_cell_pos
    float dwv[3][3];
    if (PB) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float pcp = fs(fa(i2f(sc.cell[k]), sc.f[k]), 0.5f);
#pragma unroll
            for (int o = 0; o < 3; o++) offs[k][o] = fs(i2f(sc.cell[k] + o - 1), pcp);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int a = 0; a < 3; a++) dwv[k][a] = dwk(k, sc.f[a]);
    }
    const float4* row = vel + (l0[2] * H + l0[1]) * H + l0[0];
    if (PB) {
        // the same sums in paired form: (nv0, nv1), (G[3c], G[3c+1]) per
        // column c, (G[2], G[5]); nv2 and G[8] scalar
        float2 nv01 = make_float2(0.f, 0.f), g01[3], g25 = make_float2(0.f, 0.f);
        float nv2 = 0.f, g8 = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) g01[c] = make_float2(0.f, 0.f);
#pragma unroll
        for (int oz = 0; oz < 3; oz++)
#pragma unroll
            for (int oy = 0; oy < 3; oy++) {
                float wxy[3];
#pragma unroll
                for (int ox = 0; ox < 3; ox++) wxy[ox] = fm(sc.w[ox][0], sc.w[oy][1]);
#pragma unroll
                for (int ox = 0; ox < 3; ox++) {
                    float4 c4 = row[(oz * H + oy) * H + ox];
                    const float wgt = fm(wxy[ox], sc.w[oz][2]);
                    const float2 w2 = dup2(wgt), cv01 = make_float2(c4.x, c4.y);
                    nv01 = ff2(w2, cv01, nv01);
                    nv2 = ff(wgt, c4.z, nv2);
                    const float2 wv01 = fm2(w2, cv01);
                    const float wv2 = fm(wgt, c4.z);
                    const float dist[3] = {offs[0][ox], offs[1][oy], offs[2][oz]};
#pragma unroll
                    for (int c = 0; c < 3; c++) g01[c] = ff2(wv01, dup2(dist[c]), g01[c]);
                    g25 = ff2(dup2(wv2), make_float2(dist[0], dist[1]), g25);
                    g8 = ff(wv2, dist[2], g8);
                }
            }
        nv[0] = nv01.x; nv[1] = nv01.y; nv[2] = nv2;
#pragma unroll
        for (int c = 0; c < 3; c++) { G[3 * c] = g01[c].x; G[3 * c + 1] = g01[c].y; }
        G[2] = g25.x; G[5] = g25.y; G[8] = g8;
        return;
    }
#pragma unroll
    for (int oz = 0; oz < 3; oz++)
#pragma unroll
        for (int oy = 0; oy < 3; oy++) {
            float wxy[3];
#pragma unroll
            for (int ox = 0; ox < 3; ox++) wxy[ox] = fm(sc.w[ox][0], sc.w[oy][1]);
#pragma unroll
            for (int ox = 0; ox < 3; ox++) {
                float4 c4 = row[(oz * H + oy) * H + ox];
                float cv[3] = {c4.x, c4.y, c4.z};
                float wgt = fm(wxy[ox], sc.w[oz][2]);
#pragma unroll
                for (int k = 0; k < 3; k++) nv[k] = ff(wgt, cv[k], nv[k]);
                if (!PB) {
                    float g[3];
                    g[0] = fm(fm(dwv[ox][0], sc.w[oy][1]), sc.w[oz][2]);
                    g[1] = fm(fm(sc.w[ox][0], dwv[oy][1]), sc.w[oz][2]);
                    g[2] = fm(wxy[ox], dwv[oz][2]);
#pragma unroll
                    for (int col = 0; col < 3; col++)
#pragma unroll
                        for (int r = 0; r < 3; r++) G[col * 3 + r] = ff(g[col], cv[r], G[col * 3 + r]);
                } else {
                    float wv[3] = {fm(wgt, cv[0]), fm(wgt, cv[1]), fm(wgt, cv[2])};
                    float dist[3] = {offs[0][ox], offs[1][oy], offs[2][oz]};
#pragma unroll
                    for (int col = 0; col < 3; col++)
#pragma unroll
                        for (int r = 0; r < 3; r++) G[col * 3 + r] = ff(wv[r], dist[col], G[col * 3 + r]);
                }
            }
        }
}

template <bool PB>
__device__ __forceinline__ void g2p_finish(const SceneDev& S, const float* nv, const float* G, float* vel, float* dxp,
                                           float* D) {
#pragma unroll
    for (int k = 0; k < 3; k++) { vel[k] = nv[k]; dxp[k] = fm(nv[k], S.dt); }
    if (!PB) {
#pragma unroll
        for (int i = 0; i < 9; i++) D[i] = fm(G[i], S.dt);
    } else {
#pragma unroll
        for (int i = 0; i < 9; i++) D[i] = fm(fm(G[i], S.dt), 4.0f);
    }
}

// Interaction force at grid cell cc (pbmpm.wgsl:104-134), added to f.
__device__ __noinline__ void interaction_force(const SceneDev& S, const int* cc, float* f) {
    float dv[3] = {fs(i2f(cc[0]), S.ipos[0]), fs(i2f(cc[1]), S.ipos[1]), fs(i2f(cc[2]), S.ipos[2])};
    float dist = len3(dv);
    if (!(dist < S.irad)) return;
    float pd[3] = {0.f, 0.f, 1.f};
    float l = len3(dv);
    if (l > 0.001f) {
#pragma unroll
        for (int k = 0; k < 3; k++) pd[k] = fd(dv[k], l);
    }
    float fl = fd(dist, S.irad);
    float falloff = fs(1.0f, fm(fl, fl));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float af = (S.imode == 0u) ? fm(fm(pd[k], S.istr), falloff)
                                   : fm(fm(fm(-pd[k], S.istr), falloff), fs(1.0f, falloff));
        f[k] = fa(f[k], af);
    }
}

// i32((x * RN(1/dt)) * scale) and i32((x * dt) * scale), folded into one
// product when the scale is a power of two (SceneDev::fold)
template <bool FOLD>
__device__ __forceinline__ int32_t enc_rdt(const SceneDev& S, float x) {
    return FOLD ? f2i(fm(x, S.rdts)) : f2i(fm(fm(x, S.rdt), S.scale));
}
template <bool FOLD>
__device__ __forceinline__ int32_t enc_dt(const SceneDev& S, float x) {
    return FOLD ? f2i(fm(x, S.dts)) : f2i(fm(fm(x, S.dt), S.scale));
}

// The force over a cell that the particle-side force term uses (pbmpm.wgsl:104-137),
// divided by the force divisor.
__device__ __forceinline__ void cell_force(const SceneDev& S, const int* cc, float* fo) {
    if (S.iact != 0u) {
        float f3[3] = {S.g[0], S.g[1], S.g[2]};
        interaction_force(S, cc, f3);
#pragma unroll
        for (int k = 0; k < 3; k++) fo[k] = fm(f3[k], S.rfdiv);
    } else {
#pragma unroll
        for (int k = 0; k < 3; k++) fo[k] = S.gdiv[k];
    }
}

// Interaction scenes: the cells' forces are formed once per tile, into three
// f32 planes of shared memory, except at edge 16 (no room: per particle).
template <int E> __host__ __device__ constexpr bool force_table() { return E < 16; }

// affine P2G + particle-side forces (pbmpm.wgsl:41-147) into the shared tile,
// of the first transfer.  Within one substep positions and masses do not change
// between PBMPM iterations, so every iteration's mass sums and force sums equal
// this transfer's: only it adds the masses (plane 0) and the forces, and the
// caller carries both over.  NF: the force planes behind the momentum planes
// -- 0, no iteration follows: the forces go into the momentum; 1, gravity
// along S.faxis; 3, a force per axis and cell.  The i32 adds commute, so the
// cells are visited in any order: (x, y) pairs outside, z inside, sharing the
// partial affine sums of each pair.  Components 0 and 1 in paired form,
// component 2 scalar.  Without the forces an iteration's particle has 27 to 81
// products, conversions and adds less, and no call of the interaction force
// (its square roots and divisions): PBMPM, set + 4 substeps + get, 262,144
// particles with gravity 1,045 -> 955 us, 20,011 with the interaction force
// 274 -> 118 us; 4,194,304 particles, one substep, 5,464 -> 5,393 us.
template <int E, int NF, bool FOLD>
__device__ __forceinline__ void p2g_first_particle(const SceneDev& S, const TileCtx<E>& T, const Stencil& sc,
                                                   float mass, const float* dxp, const float* D, uint32_t* acc) {
    constexpr int H = E + 2, NC = H * H * H, MOM = 1, FRC = MOM + 3;
    int l0[3];
    bool inside = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        l0[k] = sc.cell[k] - T.origin[k];
        inside = inside && l0[k] >= 0 && l0[k] < E;
    }
    if (!inside) return;
    float off[3][3];  // off[axis][o] = (cell + o - 1) - particle_cell_pos
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float pcp = fs(fa(i2f(sc.cell[a]), sc.f[a]), 0.5f);
#pragma unroll
        for (int o = 0; o < 3; o++) off[a][o] = fs(i2f(sc.cell[a] + o - 1), pcp);
    }
    // a force component that is zero for every cell adds i32(0) = 0
    bool fon[3];
#pragma unroll
    for (int k = 0; k < 3; k++) fon[k] = NF == 0 && S.gdiv[k] != 0.0f;
    const float gax = NF == 1 ? S.gdiv[S.faxis] : 0.0f;
    uint32_t* base = acc + (l0[2] * H + l0[1]) * H + l0[0];
    const float2 D01 = make_float2(D[0], D[1]), D34 = make_float2(D[3], D[4]), D67 = make_float2(D[6], D[7]);
    const float2 dxp01 = make_float2(dxp[0], dxp[1]);
#pragma unroll
    for (int oy = 0; oy < 3; oy++)
#pragma unroll(FOLD ? 3 : 1)
        for (int ox = 0; ox < 3; ox++) {
            // aff[r] = fma(D[2][r], off_z, fma(D[1][r], off_y, D[0][r] * off_x))
            const float2 pxy01 = ff2(D34, dup2(off[1][oy]), fm2(D01, dup2(off[0][ox])));
            const float pxy2 = ff(D[5], off[1][oy], fm(D[2], off[0][ox]));
            const float wxy = fm(sc.w[ox][0], sc.w[oy][1]);
#pragma unroll
            for (int oz = 0; oz < 3; oz++) {
                const float wgt = fm(wxy, sc.w[oz][2]);
                const float wm = fm(wgt, mass);
                const float2 aff01 = ff2(D67, dup2(off[2][oz]), pxy01);
                const float aff2 = ff(D[8], off[2][oz], pxy2);
                const float2 m01 = fm2(dup2(wm), fa2(dxp01, aff01));
                const float m2 = fm(wm, fa(dxp[2], aff2));
                uint32_t v[3];
                if (FOLD) {
                    const float2 x01 = fm2(m01, dup2(S.rdts));
                    v[0] = (uint32_t)f2i(x01.x);
                    v[1] = (uint32_t)f2i(x01.y);
                } else {
                    v[0] = (uint32_t)enc_rdt<FOLD>(S, m01.x);
                    v[1] = (uint32_t)enc_rdt<FOLD>(S, m01.y);
                }
                v[2] = (uint32_t)enc_rdt<FOLD>(S, m2);
                uint32_t* cell = base + (oz * H + oy) * H + ox;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    if (fon[k]) v[k] += (uint32_t)enc_dt<FOLD>(S, fm(S.gdiv[k], wm));
                    atomicAdd(cell + (MOM + k) * NC, v[k]);
                }
                atomicAdd(cell, (uint32_t)f2i(fm(wm, S.scale)));
                if (NF == 1) atomicAdd(cell + FRC * NC, (uint32_t)enc_dt<FOLD>(S, fm(gax, wm)));
                if (NF == 3) {
                    float fo[3];
                    if (force_table<E>()) {
                        const float* ft = reinterpret_cast<const float*>(cell) + (FRC + 3) * NC;
#pragma unroll
                        for (int k = 0; k < 3; k++) fo[k] = ft[k * NC];
                    } else {
                        const int cc[3] = {sc.cell[0] + ox - 1, sc.cell[1] + oy - 1, sc.cell[2] + oz - 1};
                        cell_force(S, cc, fo);
                    }
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        atomicAdd(cell + (FRC + k) * NC, (uint32_t)enc_dt<FOLD>(S, fm(fo[k], wm)));
                }
            }
        }
}

// Affine P2G of momentum only, of the iterations.  Cells go in pairs (FFMA2 /
// FMUL2): for each y, the cells x = 0, 1 of every z, the cells z = 0, 1 at
// x = 2, and one single cell.  13 of 27 cells' products come for free, where
// pairs of components left every third one single: 262,144 particles, set + 4
// substeps + get, 953 -> 931 us.
template <int E, bool FOLD>
__device__ __forceinline__ void p2g_iter_particle(const SceneDev& S, const TileCtx<E>& T, const Stencil& sc,
                                                  float mass, const float* dxp, const float* D, uint32_t* acc) {
    constexpr int H = E + 2, NC = H * H * H;
    int l0[3];
    bool inside = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        l0[k] = sc.cell[k] - T.origin[k];
        inside = inside && l0[k] >= 0 && l0[k] < E;
    }
    if (!inside) return;
    float off[3][3];  // off[axis][o] = (cell + o - 1) - particle_cell_pos
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float pcp = fs(fa(i2f(sc.cell[a]), sc.f[a]), 0.5f);
#pragma unroll
        for (int o = 0; o < 3; o++) off[a][o] = fs(i2f(sc.cell[a] + o - 1), pcp);
    }
    uint32_t* base = acc + (l0[2] * H + l0[1]) * H + l0[0];
    const float2 wx01 = make_float2(sc.w[0][0], sc.w[1][0]), offx01 = make_float2(off[0][0], off[0][1]);
    auto pair = [&](const float2* p, float2 wxy, float2 wz, float2 oz, uint32_t* ca, uint32_t* cb) {
        const float2 wm = fm2(fm2(wxy, wz), dup2(mass));
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float2 m = fm2(wm, fa2(dup2(dxp[k]), ff2(dup2(D[6 + k]), oz, p[k])));
            m = FOLD ? fm2(m, dup2(S.rdts)) : fm2(fm2(m, dup2(S.rdt)), dup2(S.scale));
            atomicAdd(ca + k * NC, (uint32_t)f2i(m.x));
            atomicAdd(cb + k * NC, (uint32_t)f2i(m.y));
        }
    };
#pragma unroll
    for (int oy = 0; oy < 3; oy++) {
        const float wy = oy == 0 ? sc.w[0][1] : (oy == 1 ? sc.w[1][1] : sc.w[2][1]);
        const float offy = oy == 0 ? off[1][0] : (oy == 1 ? off[1][1] : off[1][2]);
        float2 p01[3], p22[3];
        float p2[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            // aff[k] = fma(D[2][k], off_z, fma(D[1][k], off_y, D[0][k] * off_x))
            p01[k] = ff2(dup2(D[3 + k]), dup2(offy), fm2(dup2(D[k]), offx01));
            p2[k] = ff(D[3 + k], offy, fm(D[k], off[0][2]));
            p22[k] = dup2(p2[k]);
        }
        const float2 wxy01 = fm2(wx01, dup2(wy));
        const float wxy2 = fm(sc.w[2][0], wy);
        uint32_t* row = base + oy * H;
#pragma unroll
        for (int oz = 0; oz < 3; oz++)
            pair(p01, wxy01, dup2(sc.w[oz][2]), dup2(off[2][oz]), row + oz * H * H, row + oz * H * H + 1);
        pair(p22, dup2(wxy2), make_float2(sc.w[0][2], sc.w[1][2]), make_float2(off[2][0], off[2][1]), row + 2,
             row + H * H + 2);
        const float wm = fm(fm(wxy2, sc.w[2][2]), mass);
#pragma unroll
        for (int k = 0; k < 3; k++)
            atomicAdd(row + 2 * H * H + 2 + k * NC,
                      (uint32_t)enc_rdt<FOLD>(S, fm(wm, fa(dxp[k], ff(D[6 + k], off[2][2], p2[k])))));
    }
}

template <int E>
__device__ __forceinline__ void flush_tile(uint32_t* acc, int4* dst) {
    constexpr int H = E + 2, NC = H * H * H;
    for (int j = threadIdx.x; j < NC; j += blockDim.x)
        dst[j] = make_int4((int)acc[j], (int)acc[NC + j], (int)acc[2 * NC + j], (int)acc[3 * NC + j]);
}

// the first PBMPM transfer's tile: the forces join the momentum, and their
// planes go to tiles_f for the iterations
template <int E, int NF>
__device__ __forceinline__ void flush_first(const uint32_t* acc, uint32_t axis, int4* dst, uint32_t* frc) {
    constexpr int H = E + 2, NC = H * H * H;
    for (int j = threadIdx.x; j < NC; j += blockDim.x) {
        uint32_t m[3] = {acc[NC + j], acc[2 * NC + j], acc[3 * NC + j]};
#pragma unroll
        for (int k = 0; k < NF; k++) {
            const uint32_t f = acc[(4 + k) * NC + j];
            if (NF == 1) {
#pragma unroll
                for (int a = 0; a < 3; a++) m[a] += axis == (uint32_t)a ? f : 0u;
            } else {
                m[k] += f;
            }
            if (frc != nullptr) frc[k * NC + j] = f;
        }
        dst[j] = make_int4((int)acc[j], (int)m[0], (int)m[1], (int)m[2]);
    }
}

// Momentum accumulator of the PBMPM iterations, 3 planes x (E+2)^3: the planes
// start at the tile's force sums (bulk copies that complete on fc) and at 0
// where no force plane exists.  Returns with the copies in flight.
template <int E>
__device__ __forceinline__ void start_mom(const Ctx& c, uint32_t st, uint32_t axis, uint32_t* acc, HaloCopy& fc) {
    constexpr int H = E + 2, NC = H * H * H;
    const bool one = c.force_planes == 1u;
    if (threadIdx.x == 0) {
        // the previous tile's accumulators were read through the generic proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const uint32_t n = one ? 1u : 3u;
        const uint32_t* src = c.tiles_f + (size_t)st * n * NC;
        mbar_expect_tx(fc.mbar, n * NC * 4u);
        for (uint32_t k = 0; k < n; k++) bulk_g2s(acc + (one ? axis : k) * NC, src + (size_t)k * NC, NC * 4u, fc.mbar);
    }
    if (!one) return;
    const uint32_t a = axis == 0u ? 1u : 0u, b = axis == 2u ? 1u : 2u;
    uint4* pa = reinterpret_cast<uint4*>(acc + a * NC);
    uint4* pb = reinterpret_cast<uint4*>(acc + b * NC);
    for (int j = threadIdx.x; j < NC / 4; j += blockDim.x) {
        pa[j] = make_uint4(0u, 0u, 0u, 0u);
        pb[j] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// halo record of a PBMPM iteration: the cell's reciprocal mass RN(1/m) of the
// substep (the same in every tile that covers the cell) in the mass word,
// this tile's momentum sums in the other three
template <int E>
__device__ __forceinline__ void flush_mom(const uint32_t* acc, const float* rm_s, int4* dst) {
    constexpr int H = E + 2, NC = H * H * H;
#pragma unroll 4
    for (int j = threadIdx.x; j < NC; j += blockDim.x)
        dst[j] = make_int4(__float_as_int(rm_s[j]), (int)acc[j], (int)acc[NC + j], (int)acc[2 * NC + j]);
}

// PLANES accumulator planes x (E+2)^3
template <int E, int PLANES = 4>
__device__ __forceinline__ void zero_acc(uint32_t* acc) {
    constexpr int H = E + 2, NC = H * H * H;
    static_assert(NC % 4 == 0, "planes of 16-byte words");
    uint4* a4 = reinterpret_cast<uint4*>(acc);
    for (int j = threadIdx.x; j < PLANES * NC / 4; j += blockDim.x) a4[j] = make_uint4(0u, 0u, 0u, 0u);
}

// A halo copy wait ran out: report it, give the copies in flight a second
// bounded wait (so no bulk write lands after the CTA has exited), and let the
// caller return.  fc: the accumulators' copy of the PBMPM iterations, whose
// own wait comes after (its parity still names the phase in flight).
__device__ __noinline__ void copy_wait_failed(const Ctx& c, HaloCopy& hc, HaloCopy* fc = nullptr) {
    if (threadIdx.x == 0) {
        atomicOr(&c.counters->status, ST_COPY_TIMEOUT);
        mbar_wait_parity(hc.mbar, hc.parity ^ 1u, COPY_WAIT_LIMIT);
        if (fc != nullptr) mbar_wait_parity(fc->mbar, fc->parity, COPY_WAIT_LIMIT);
    }
    __syncthreads();
}

__device__ __forceinline__ uint32_t n_tiles_now(const Ctx& c) {
    uint32_t n = c.counters->n_st;
    return n < c.max_tiles ? n : c.max_tiles;
}

// Tile scheduling of the persistent tile kernels: CTA b takes claim slot b
// first, then the next unclaimed slot (gridDim.x + ticket) each time it
// finishes a tile, so CTAs with light tiles take more of them and a launch
// ends within about one tile of the average.  Slot k maps to a tile through
// tile_order (Morton order, so the tiles in flight at one time are neighbours
// and share their halo data in L2; read from its end on alternate launches,
// so a launch starts on the tiles the previous one wrote last).  Each tile's
// results go to its own slots, so which CTA runs a tile, and when, changes
// nothing in them.  Returns n (stop) past the last slot.
__device__ __forceinline__ uint32_t tile_at(const Ctx& c, uint32_t k, uint32_t n) {
    if (k >= n) return n;
    if (!c.tile_order) return k;
    const uint32_t st = __ldg(c.tile_order + (c.order_rev ? n - 1u - k : k));
    return st < n ? st : n;
}

// Called by thread 0; the caller broadcasts the result through shared memory.
__device__ __forceinline__ uint32_t claim_tile(const Ctx& c, uint32_t n) {
    return tile_at(c, gridDim.x + atomicAdd(&c.counters->tile_ticket, 1u), n);
}

// Claim order of the tiles: a counting sort in one CTA by a 12- or 15-bit
// Morton bucket of the tile coordinates (4 or 5 low bits per axis, offset per
// scene), so the tiles of a 16^3- or 32^3-tile neighbourhood are ordered along
// the Morton curve (tiles in one bucket keep an arbitrary order).  The scatter
// positions are the buckets' prefix offsets, so the result is always a
// permutation.
constexpr uint32_t TILE_ORDER_BUCKETS = 1u << 15;   // the wider bucket count
constexpr size_t TILE_ORDER_SMEM = TILE_ORDER_BUCKETS * 4;   // 4 bits per axis: an eighth of it
constexpr uint32_t TILE_ORDER_MIN = 256;    // at most this many tiles keep the compact order

__device__ __forceinline__ uint32_t spread3_5(uint32_t v) {
    uint32_t x = v & 31u;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// bucket of a tile key: the Morton code of the low `bits` bits of each
// coordinate (bits = 4 or 5), offset per scene, modulo nb = 2^(3 bits)
__device__ __forceinline__ uint32_t tile_bucket(uint64_t key, uint32_t axis_mask, uint32_t nb) {
    const uint32_t m = spread3_5((uint32_t)(key >> 32) & axis_mask) |
                       (spread3_5((uint32_t)(key >> 16) & axis_mask) << 1) |
                       (spread3_5((uint32_t)key & axis_mask) << 2);
    return (m + (uint32_t)(key >> 48) * 0x9E3779B1u) & (nb - 1u);
}

template <uint32_t BITS>
__device__ __forceinline__ void tile_order_sort(const Ctx& c, uint32_t n, uint32_t* hist, uint32_t* warp_sum) {
    constexpr uint32_t NB = 1u << (3 * BITS), PER = NB / 1024u;   // buckets, buckets per thread
    constexpr uint32_t AXIS = (1u << BITS) - 1u;
    for (uint32_t b = threadIdx.x; b < NB; b += 1024) hist[b] = 0u;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 1024) atomicAdd(&hist[tile_bucket(c.st_key[i], AXIS, NB)], 1u);
    __syncthreads();
    // exclusive prefix sums: each thread scans its PER consecutive buckets,
    // the thread totals are scanned across the block
    const uint32_t b0 = threadIdx.x * PER;
    uint32_t tot = 0;
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) tot += hist[b0 + k];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = tot;
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += v;
    }
    if (lane == 31u) warp_sum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = warp_sum[lane], wi = w;
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, wi, d);
            if (lane >= d) wi += v;
        }
        warp_sum[lane] = wi - w;   // exclusive over warps
    }
    __syncthreads();
    uint32_t run = warp_sum[warp] + inc - tot;
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) {
        const uint32_t h = hist[b0 + k];
        hist[b0 + k] = run;
        run += h;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 1024) {
        const uint32_t pos = atomicAdd(&hist[tile_bucket(c.st_key[i], AXIS, NB)], 1u);
        if (pos < n) c.tile_order[pos] = i;
    }
}

// A CTA leaves a tile kernel: the last one to leave zeroes the ticket for the
// next launch (every CTA has claimed its last ticket before it counts itself).
__device__ __forceinline__ void tiles_done(const Ctx& c) {
    if (threadIdx.x == 0) {
        if (atomicAdd(&c.counters->tile_done, 1u) == gridDim.x - 1u) {
            c.counters->tile_ticket = 0u;
            c.counters->tile_done = 0u;
        }
    }
}

// Exclusive scan of the tiles' particle counts (compact order) by one CTA of
// 1024 threads, four tiles per thread and pass, into st_begin / st_count and
// the slots' offsets; returns the total.
__device__ __forceinline__ uint32_t plan_offsets(const Ctx& c, uint32_t n, uint32_t* warp_sum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < n; base += 4096u) {
        const uint32_t i0 = base + threadIdx.x * 4u;
        uint32_t slot[4], cnt[4], tot = 0;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) slot[k] = i0 + k < n ? c.st_slot[i0 + k] : INVALID;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            cnt[k] = slot[k] != INVALID ? c.slot_count[slot[k]] : 0u;
            tot += cnt[k];
        }
        uint32_t inc = tot;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += v;
        }
        if (lane == 31u) warp_sum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            uint32_t wi = warp_sum[lane];
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, wi, d);
                if (lane >= d) wi += v;
            }
            warp_sum[lane] = wi;   // inclusive over warps
        }
        __syncthreads();
        uint32_t off = carry + (warp ? warp_sum[warp - 1u] : 0u) + inc - tot;
        carry += warp_sum[31];
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            if (slot[k] != INVALID) {
                c.slot_off[slot[k]] = off;
                c.st_begin[i0 + k] = off;
                c.st_count[i0 + k] = cnt[k];
                off += cnt[k];
            }
        __syncthreads();
    }
    return carry;
}

// Everything the tile kernels need beside the sorted particles, in one launch
// after bin_insert.  CTA 0: particle offsets of the tiles, the substep's
// counters, the claim order of the tiles.  The other CTAs: neighbour table of
// the compact tiles -- entry st*27 + d is the compact index of the tile at
// offset d = 9(dz+1) + 3(dy+1) + (dx+1), or -1 when that tile is unoccupied or
// past the tile storage.  Latency-bound (two dependent gathers and a scan over
// the occupied tiles).  The tiles are numbered as bin_insert claims them, so
// no pass scans the hash table: this launch, bin_scatter (which empties the
// table) and bin_insert replace eight (clear, three compaction passes over
// every table slot, neighbour table, claim order).
template <int E>
__global__ void __launch_bounds__(1024) k_bin_plan(Ctx c) {
    const uint32_t n_all = c.counters->n_ins;
    const uint32_t n = n_all < c.max_tiles ? n_all : c.max_tiles;
    if (blockIdx.x > 0) {
        const uint32_t n27 = n * 27u;
        for (uint32_t i = (blockIdx.x - 1u) * 1024u + threadIdx.x; i < n27; i += (gridDim.x - 1u) * 1024u) {
            uint32_t st = i / 27u, d = i - st * 27u;
            int r = (int)st;
            if (d != 13u) {
                uint32_t scene;
                int sx, sy, sz;
                unpack_key(c.st_key[st], scene, sx, sy, sz);
                sx += (int)(d % 3u) - 1;
                sy += (int)((d / 3u) % 3u) - 1;
                sz += (int)(d / 9u) - 1;
                uint32_t slot = tile_lookup(c, pack_key(scene, sx, sy, sz), scene, sx, sy, sz);
                r = (slot == INVALID) ? -1 : (int)c.slot_st[slot];
                if (r >= (int)c.max_tiles) r = -1;
            }
            c.st_nbr[i] = r;
        }
        return;
    }
    extern __shared__ uint4 smem_raw[];
    uint32_t* hist = reinterpret_cast<uint32_t*>(smem_raw);
    __shared__ uint32_t warp_sum[32];
    const uint32_t total = plan_offsets(c, n_all, warp_sum);
    if (threadIdx.x == 0) {
        Counters* k = c.counters;
        k->n_st = n_all;
        k->n_binned = total;
        if (n_all > c.max_tiles) atomicOr(&k->status, ST_TILE_OVERFLOW);
        k->n_plast = 0u;
        k->n_col = 0u;
        k->step += c.step_inc;
        k->tile_ticket = 0u;
        k->tile_done = 0u;
        k->n_carry = 0u;
    }
    if (!c.tile_order) return;
    uint32_t mode = c.order_mode;
    // automatic: few tiles nearly all run at once, so their order gains
    // nothing; up to 4,096 tiles 4 bits per axis (4,096 buckets), else 5 (32,768)
    if (mode != 1u && mode != 4u && mode != 5u) mode = n <= TILE_ORDER_MIN ? 1u : (n <= 4096u ? 4u : 5u);
    if (mode == 5u && c.order_bits < 5u) mode = 4u;
    if (mode == 1u) {
        for (uint32_t i = threadIdx.x; i < n; i += 1024) c.tile_order[i] = i;
        return;
    }
    if (mode == 4u) tile_order_sort<4>(c, n, hist, warp_sum);
    else tile_order_sort<5>(c, n, hist, warp_sum);
}

// CTA widths of the tile kernels and the registers a thread may use.  Every
// tile kernel is bound by issue and latency (IPC 1.2 to 2.1 of 4), so warps
// count for more than registers until the compiler spills: explicit P2G and
// both G2Ps run 24 warps per SM at 80 registers (P2G without spills, G2P with
// about 80 bytes) where shared memory allows three CTAs of 256, against 16 at
// 99 to 128: 1,000,003 explicit particles at edge 8, set + 4 substeps + get,
// 778 -> 700 us.  At 64 registers the G2Ps spill 200 bytes and lose it again.
// At edge 16 two CTAs (93 KB of halo sums each) fit: explicit P2G 384 threads
// at 80 registers (117 -> 109 us for 1,000,003 particles at 0.6 per cell),
// the G2Ps 320 at 96 (142 -> 133 us, PBMPM 221 -> 211 us for 1.5 M).
constexpr int max_regs(int bs, int regs) { return 65536 / (regs * bs) > 0 ? 65536 / (regs * bs) : 1; }
template <int E> constexpr int tile_block() { return E == 4 ? 128 : 256; }
template <int E> constexpr int p2g_block() { return E == 16 ? 384 : tile_block<E>(); }
template <int E> constexpr int g2p_block() { return E == 16 ? 320 : tile_block<E>(); }
template <int E> constexpr int iter_block() { return E == 16 ? 512 : E == 12 ? 320 : tile_block<E>(); }
// few tiles: wider CTAs at the two smallest edges, where a launch lasts about
// as long as its heaviest tile
template <int E> constexpr int wide_block() { return E == 8 ? 512 : E == 4 ? 256 : 0; }
// The iterations (32 KB of shared memory per CTA at edge 8) spill 60 to 140
// bytes at 80 registers, and 24 warps still beat 16: 524,288 particles at edge
// 8, set + 2 substeps + get, 834 -> 764 us.  32 warps at 64 registers lose it
// (791 us), as do 24 warps in one CTA of 768 (edge 8 with few tiles 955 -> 994
// us; edge 16 with 4.2 M particles 5,393 -> 5,788 us), 640 threads at edge 16
// (5,616 us) and 80 registers at edge 4 (118 -> 120 us).  At edge 12 shared
// memory holds two CTAs: 320 threads at 96 registers 5,017 us for 4.2 M particles,
// 256 at 128 5,090, 384 at 80 5,537; the other passes at 384 lose 3 %.
constexpr int iter_regs(int e, int bs) { return e == 8 && bs == 256 ? 80 : e == 12 ? 96 : 128; }
constexpr int p2g_regs(int bs) { return bs >= 512 ? 128 : 80; }
constexpr int g2p_regs(int bs) { return bs >= 512 ? 128 : bs == 320 ? 96 : 80; }
// The first PBMPM transfer has NF force planes behind its four: at edge 16 one
// CTA fits beside them, and 768 threads bring its 24 warps.
template <int E, int NF> constexpr int first_block() { return E == 16 && NF > 0 ? 768 : tile_block<E>(); }
constexpr int first_regs(int e, int bs, int nf) { return (e == 16 && nf == 0) || bs == 512 ? 128 : 80; }
template <int E, int NF> constexpr size_t first_smem() {
    return (size_t)(E + 2) * (E + 2) * (E + 2) * (size_t)(16 + 4 * NF + (NF == 3 && force_table<E>() ? 12 : 0));
}

// ------------------------------------------------------------------
// explicit P2G (particleToGrid.cs.wgsl:27-79)
// ------------------------------------------------------------------
// 27-cell scatter of mass, momentum and stress force.  Cells go in pairs
// (FFMA2 / FMUL2) as in p2g_iter_particle: 1,000,003 particles, set + 4
// substeps + get, 698 -> 684 us (the scatter issues a third less, and latency
// takes most of it back).
template <int E>
__device__ __forceinline__ void scatter_explicit(const SceneDev& S, const Stencil& sc, float mass, const float* pm,
                                                 const float* M, uint32_t* base) {
    constexpr int H = E + 2, NC = H * H * H;
    const float2 wx01 = make_float2(sc.w[0][0], sc.w[1][0]);
    const float2 dwx01 = make_float2(dwk(0, sc.f[0]), dwk(1, sc.f[0]));
    const float wx2 = sc.w[2][0], dwx2 = dwk(2, sc.f[0]);
    const float wz[3] = {sc.w[0][2], sc.w[1][2], sc.w[2][2]};
    const float dwz[3] = {dwk(0, sc.f[2]), dwk(1, sc.f[2]), dwk(2, sc.f[2])};
    // a = dwx wy, b = wx dwy, c = wx wy of the two cells
    auto pair = [&](float2 a, float2 b, float2 cc, float2 wz2, float2 dwz2, uint32_t* c0, uint32_t* c1) {
        const float2 w2 = fm2(cc, wz2);
        const float2 g0 = fm2(fm2(a, wz2), dup2(S.rcd[0]));
        const float2 g1 = fm2(fm2(b, wz2), dup2(S.rcd[1]));
        const float2 g2 = fm2(fm2(cc, dwz2), dup2(S.rcd[2]));
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float2 sf = ff2(dup2(M[6 + k]), g2, ff2(dup2(M[3 + k]), g1, fm2(dup2(M[k]), g0)));
            const float2 x = fm2(ff2(w2, dup2(pm[k]), fm2(sf, dup2(S.dt))), dup2(S.scale));
            atomicAdd(c0 + (k + 1) * NC, (uint32_t)f2i(x.x));
            atomicAdd(c1 + (k + 1) * NC, (uint32_t)f2i(x.y));
        }
        const float2 m2 = fm2(fm2(w2, dup2(mass)), dup2(S.scale));
        atomicAdd(c0, (uint32_t)f2i(m2.x));
        atomicAdd(c1, (uint32_t)f2i(m2.y));
    };
#pragma unroll 1
    for (int oy = 0; oy < 3; oy++) {
        const float wy = oy == 0 ? sc.w[0][1] : (oy == 1 ? sc.w[1][1] : sc.w[2][1]);
        const float dwy = oy == 0 ? dwk(0, sc.f[1]) : (oy == 1 ? dwk(1, sc.f[1]) : dwk(2, sc.f[1]));
        const float2 a01 = fm2(dwx01, dup2(wy)), b01 = fm2(wx01, dup2(dwy)), c01 = fm2(wx01, dup2(wy));
        const float a2 = fm(dwx2, wy), b2 = fm(wx2, dwy), c2 = fm(wx2, wy);
        uint32_t* row = base + oy * H;
#pragma unroll
        for (int oz = 0; oz < 3; oz++)
            pair(a01, b01, c01, dup2(wz[oz]), dup2(dwz[oz]), row + oz * H * H, row + oz * H * H + 1);
        pair(dup2(a2), dup2(b2), dup2(c2), make_float2(wz[0], wz[1]), make_float2(dwz[0], dwz[1]), row + 2,
             row + H * H + 2);
        const float wgt = fm(c2, wz[2]);
        const float g[3] = {fm(fm(a2, wz[2]), S.rcd[0]), fm(fm(b2, wz[2]), S.rcd[1]), fm(fm(c2, dwz[2]), S.rcd[2])};
        float sf[3];
        mv3(M, g, sf);
        uint32_t* cell = row + 2 * H * H + 2;
#pragma unroll
        for (int k = 0; k < 3; k++)
            atomicAdd(cell + (k + 1) * NC, (uint32_t)f2i(fm(ff(wgt, pm[k], fm(sf[k], S.dt)), S.scale)));
        atomicAdd(cell, (uint32_t)f2i(fm(fm(wgt, mass), S.scale)));
    }
}

template <int E, int BS>
__global__ void __launch_bounds__(BS, max_regs(BS, p2g_regs(BS))) k_p2g_explicit(Ctx c) {
    constexpr int H = E + 2, NC = H * H * H;
    extern __shared__ uint4 smem_raw[];
    uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);
    __shared__ SceneDev S;
    __shared__ uint32_t s_next;
    uint32_t cur_scene = INVALID;
    uint32_t n_st = n_tiles_now(c);
    for (uint32_t st = tile_at(c, blockIdx.x, n_st); st < n_st; st = s_next) {
        TileCtx<E> T;
        Feed<BS, 6, true> feed;
        feed.begin(c.work_in, c.n_particles, c.sorted, c.st_begin[st], c.st_count[st]);
        tile_begin<E>(c, st, S, T, cur_scene);
        zero_acc<E>(acc);
        __syncthreads();
        for (; feed.more(); feed.next()) {
            float4 r[6];
            feed.take(r);
            PState p;
            unpack_particle<6>(r, feed.tail(), p);
            Stencil sc;
            make_stencil(S, p.pos, sc);
            int l0[3];
            bool inside = true;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                l0[k] = sc.cell[k] - T.origin[k];
                inside = inside && l0[k] >= 0 && l0[k] < E;
            }
            if (!inside) continue;
            float M[9];
            stress_matrix(S, p, M);
            float pm[3] = {fm(p.mass, p.vel[0]), fm(p.mass, p.vel[1]), fm(p.mass, p.vel[2])};
            scatter_explicit<E>(S, sc, p.mass, pm, M, acc + (l0[2] * H + l0[1]) * H + l0[0]);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_next = claim_tile(c, n_st);
        flush_tile<E>(acc, c.tiles_a + (size_t)st * NC);
        __syncthreads();
    }
    tiles_done(c);
}

// ------------------------------------------------------------------
// G2P + integrate (explicit: gridToParticle.cs.wgsl:28-80; PBMPM :82-130;
// integrateParticles.wgsl:14-72)
// ------------------------------------------------------------------
template <int E, bool PB, int BS, int RM = 0>
__global__ void __launch_bounds__(BS, max_regs(BS, g2p_regs(BS))) k_g2p_integrate(Ctx c) {
    extern __shared__ uint4 smem_raw[];
    int4* cell = reinterpret_cast<int4*>(smem_raw);
    const float4* vel = reinterpret_cast<const float4*>(smem_raw);
    __shared__ SceneDev S;
    __shared__ int nbr[27];
    __shared__ uint64_t mbar;
    if (threadIdx.x == 0) mbar_init1(&mbar);
    __syncthreads();
    HaloCopy hc{&mbar, 0u};
    __shared__ uint32_t s_next;
    uint32_t cur_scene = INVALID;
    uint32_t n_st = n_tiles_now(c);
    for (uint32_t st = tile_at(c, blockIdx.x, n_st); st < n_st; st = s_next) {
        TileCtx<E> T;
        const uint32_t begin = c.st_begin[st];
        Feed<BS, 6, true> feed;
        feed.begin(c.work_in, c.n_particles, c.sorted, begin, c.st_count[st]);
        tile_begin<E>(c, st, S, T, cur_scene);
        load_neighbors(c, st, nbr);
        __syncthreads();
        if (!assemble_velocity_tile<E, BS, PB, RM>(c.tiles_b, S, T, nbr, cell, hc)) {
            copy_wait_failed(c, hc);
            tiles_done(c);
            return;
        }
        __syncthreads();
        for (; feed.more(); feed.next()) {
            const uint32_t slot = begin + feed.i;
            float4 r[6];
            feed.take(r);
            PState p;
            unpack_particle<6>(r, feed.tail(), p);
            Stencil sc;
            make_stencil(S, p.pos, sc);
            float nv[3], G[9];
            g2p_gather<E, PB>(T, vel, sc, nv, G);
            g2p_finish<PB>(S, nv, G, p.vel, p.dxp, p.D);
            integrate(c, S, p, slot);
            store_particle(c.work_out, c.n_particles, slot, p);
            c.ids_out[slot] = __ldg(c.ids_in + feed.pid) & ~ID_KEEP;
        }
        if (threadIdx.x == 0) s_next = claim_tile(c, n_st);
        __syncthreads();
    }
    tiles_done(c);
}

// ------------------------------------------------------------------
// PBMPM first iteration: constraints + affine P2G + forces
// (pbmpm.wgsl:154-178); writes the iteration records
// ------------------------------------------------------------------
__device__ __forceinline__ void store_iter_rec(const Ctx& c, uint32_t t, const float* pos, float mass, const float* Fe,
                                               const float* Fei, float relax) {
    float4* r = c.iter_rec + t;
    const size_t n = c.n_particles;
    r[0] = make_float4(pos[0], pos[1], pos[2], mass);
    r[n] = make_float4(Fe[0], Fe[1], Fe[2], Fe[3]);
    r[2 * n] = make_float4(Fe[4], Fe[5], Fe[6], Fe[7]);
    r[3 * n] = make_float4(Fe[8], Fei[0], Fei[1], Fei[2]);
    r[4 * n] = make_float4(Fei[3], Fei[4], Fei[5], Fei[6]);
    r[5 * n] = make_float4(Fei[7], Fei[8], relax, 0.f);
}

__device__ __forceinline__ void unpack_iter_rec(const float4* r, float* pos, float& mass, float* Fe, float* Fei,
                                                float& relax) {
    const float4 q0 = r[0], q1 = r[1], q2 = r[2], q3 = r[3], q4 = r[4], q5 = r[5];
    pos[0] = q0.x; pos[1] = q0.y; pos[2] = q0.z; mass = q0.w;
    Fe[0] = q1.x; Fe[1] = q1.y; Fe[2] = q1.z; Fe[3] = q1.w;
    Fe[4] = q2.x; Fe[5] = q2.y; Fe[6] = q2.z; Fe[7] = q2.w;
    Fe[8] = q3.x; Fei[0] = q3.y; Fei[1] = q3.z; Fei[2] = q3.w;
    Fei[3] = q4.x; Fei[4] = q4.y; Fei[5] = q4.z; Fei[6] = q4.w;
    Fei[7] = q5.x; Fei[8] = q5.y; relax = q5.z;
}

template <int E, int BS, int NF>
__global__ void __launch_bounds__(BS, max_regs(BS, first_regs(E, BS, NF))) k_pbmpm_first(Ctx c) {
    constexpr int H = E + 2, NC = H * H * H;
    extern __shared__ uint4 smem_raw[];
    uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);
    __shared__ SceneDev S;
    __shared__ uint32_t s_next;
    uint32_t cur_scene = INVALID;
    uint32_t n_st = n_tiles_now(c);
    for (uint32_t st = tile_at(c, blockIdx.x, n_st); st < n_st; st = s_next) {
        TileCtx<E> T;
        const uint32_t begin = c.st_begin[st];
        Feed<BS, 9, true> feed;
        feed.begin(c.work_in, c.n_particles, c.sorted, begin, c.st_count[st]);
        tile_begin<E>(c, st, S, T, cur_scene);
        zero_acc<E, 4 + NF>(acc);
        __syncthreads();
        if (NF == 3 && force_table<E>()) {
            float* ft = reinterpret_cast<float*>(acc) + 7 * NC;
            for (int j = threadIdx.x; j < NC; j += BS) {
                const int cc[3] = {T.origin[0] - 1 + j % H, T.origin[1] - 1 + (j / H) % H, T.origin[2] - 1 + j / (H * H)};
                float fo[3];
                cell_force(S, cc, fo);
#pragma unroll
                for (int k = 0; k < 3; k++) ft[k * NC + j] = fo[k];
            }
            __syncthreads();
        }
        for (; feed.more(); feed.next()) {
            float4 r[9];
            feed.take(r);
            PState p;
            unpack_particle<9>(r, feed.tail(), p);
            float Fei[9];
            inv3(p.Fe, Fei);
            float relax = pbmpm_relax(S, p.Fp);
            store_iter_rec(c, begin + feed.i, p.pos, p.mass, p.Fe, Fei, relax);
            pbmpm_constraints(S, p.Fe, Fei, relax, p.D);
            Stencil sc;
            make_stencil(S, p.pos, sc);
            if (S.fold) p2g_first_particle<E, NF, true>(S, T, sc, p.mass, p.dxp, p.D, acc);
            else p2g_first_particle<E, NF, false>(S, T, sc, p.mass, p.dxp, p.D, acc);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_next = claim_tile(c, n_st);
        if (NF == 0) {
            flush_tile<E>(acc, c.tiles_a + (size_t)st * NC);
        } else {
            uint32_t* frc = c.tiles_f != nullptr ? c.tiles_f + (size_t)st * NF * NC : nullptr;
            flush_first<E, NF>(acc, S.faxis, c.tiles_a + (size_t)st * NC, frc);
        }
        __syncthreads();
    }
    tiles_done(c);
}

// PBMPM iteration i>0: G2P of iteration i-1, constraints, P2G of iteration i,
// all from the iteration records (contiguous in tile order).  Positions and
// masses are fixed within a substep, so the cell masses are the first
// transfer's: the first iteration (FIRST) forms their reciprocals from the
// mass sums; every iteration accumulates momentum only and writes, per halo
// cell, the reciprocal mass and its momentum sums, so the next pass reads the
// reciprocal masses with its own halo record.  Shared memory: the halo sums /
// velocities (16 B per cell), three momentum planes (12 B per cell) and the
// reciprocal masses (4 B per cell).
template <int E, int BS, bool FIRST>
__global__ void __launch_bounds__(BS, max_regs(BS, iter_regs(E, BS))) k_pbmpm_iter(Ctx c) {
    constexpr int H = E + 2, NC = H * H * H;
    extern __shared__ uint4 smem_raw[];
    int4* cell = reinterpret_cast<int4*>(smem_raw);
    const float4* vel = reinterpret_cast<const float4*>(smem_raw);
    uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw + NC);
    float* rm_s = reinterpret_cast<float*>(acc + 3 * NC);   // reciprocal cell masses, for the flush
    __shared__ SceneDev S;
    __shared__ int nbr[27];
    __shared__ uint64_t mbar, mbar_f;
    __shared__ uint32_t s_next;
    if (threadIdx.x == 0) {
        mbar_init1(&mbar);
        mbar_init1(&mbar_f);
    }
    __syncthreads();
    HaloCopy hc{&mbar, 0u}, fc{&mbar_f, 0u};
    uint32_t cur_scene = INVALID;
    uint32_t n_st = n_tiles_now(c);
    // a tile's own-halo copies are issued as soon as the previous tile's
    // particles are done, so they overlap that tile's flush
    const uint32_t st0 = tile_at(c, blockIdx.x, n_st);
    if (st0 < n_st)
        halo_issue<E>(c.tiles_b, st0, cell, hc);
    for (uint32_t st = st0; st < n_st; st = s_next) {
        TileCtx<E> T;
        Feed<BS, IR_PLANES, false> feed;
        feed.begin(c.iter_rec, c.n_particles, nullptr, c.st_begin[st], c.st_count[st]);
        tile_begin<E>(c, st, S, T, cur_scene);
        load_neighbors(c, st, nbr);
        start_mom<E>(c, st, __ldg(&c.scenes[T.scene].faxis), acc, fc);
        __syncthreads();
        if (!assemble_velocity_tile<E, BS, true, FIRST ? 1 : 2, true>(c.tiles_b, S, T, nbr, cell, hc,
                                                                     rm_s)) {
            copy_wait_failed(c, hc, &fc);
            tiles_done(c);
            return;
        }
        const bool fok = mbar_wait_parity(fc.mbar, fc.parity, COPY_WAIT_LIMIT);
        if (__syncthreads_or(fok ? 0 : 1)) {
            copy_wait_failed(c, hc, &fc);
            tiles_done(c);
            return;
        }
        fc.parity ^= 1u;
        for (; feed.more(); feed.next()) {
            float4 r[IR_PLANES];
            feed.take(r);
            float pos[3], mass, Fe[9], Fei[9], relax;
            unpack_iter_rec(r, pos, mass, Fe, Fei, relax);
            Stencil sc;
            make_stencil(S, pos, sc);
            float nv[3], G[9], v[3], dxp[3], D[9];
            g2p_gather<E, true>(T, vel, sc, nv, G);
            g2p_finish<true>(S, nv, G, v, dxp, D);
            pbmpm_constraints(S, Fe, Fei, relax, D);
            if (S.fold) p2g_iter_particle<E, true>(S, T, sc, mass, dxp, D, acc);
            else p2g_iter_particle<E, false>(S, T, sc, mass, dxp, D, acc);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t nx = claim_tile(c, n_st);
            s_next = nx;
            if (nx < n_st)
                halo_issue<E>(c.tiles_b, nx, cell, hc);
        }
        flush_mom<E>(acc, rm_s, c.tiles_a + (size_t)st * NC);
        __syncthreads();
    }
    tiles_done(c);
}

// ------------------------------------------------------------------
// dense grid readback for one scene (inspection only)
// ------------------------------------------------------------------
template <int E>
__global__ void __launch_bounds__(256) k_grid_dense(Ctx c, uint32_t scene, int apply_update, int4* out) {
    constexpr int H = E + 2, NC = H * H * H;
    __shared__ SceneDev S;
    __shared__ int nbr[27];
    uint32_t cur_scene = INVALID;
    uint32_t n_st = n_tiles_now(c);
    for (uint32_t st = blockIdx.x; st < n_st; st += gridDim.x) {
        TileCtx<E> T;
        tile_begin<E>(c, st, S, T, cur_scene);
        __syncthreads();
        if (T.scene != scene) continue;
        load_neighbors(c, st, nbr);
        __syncthreads();
        for (int j = threadIdx.x; j < NC; j += blockDim.x) {
            int4 s = assemble_cell<E>(c.tiles_b, nbr, j);
            if (c.tiles_m) s.x = assemble_cell<E>(c.tiles_m, nbr, j).x;
            int lx = j % H, ly = (j / H) % H, lz = j / (H * H);
            int gc[3] = {T.origin[0] - 1 + lx, T.origin[1] - 1 + ly, T.origin[2] - 1 + lz};
            if (gc[0] < 0 || gc[1] < 0 || gc[2] < 0 || gc[0] >= S.res[0] || gc[1] >= S.res[1] || gc[2] >= S.res[2]) continue;
            if (apply_update) {
                float cm = inv_s(S, s.x);
                if (cm > 0.0f) {
                    float rm = __frcp_rn(cm);
                    int32_t mi[3] = {s.y, s.z, s.w};
                    float u[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) u[k] = fa(fm(inv_s(S, mi[k]), rm), S.gdt[k]);
                    grid_bc(S, gc, u);
                    s.y = f2i(fm(fm(u[0], cm), S.scale));
                    s.z = f2i(fm(fm(u[1], cm), S.scale));
                    s.w = f2i(fm(fm(u[2], cm), S.scale));
                }
            }
            size_t o = ((size_t)gc[2] * S.res[1] + gc[1]) * S.res[0] + gc[0];
            out[o] = s;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------
// device self-test of the arithmetic helpers
// ------------------------------------------------------------------
__device__ __forceinline__ uint32_t mix32(uint64_t v) {
    v ^= v >> 33; v *= 0xff51afd7ed558ccdull; v ^= v >> 33; v *= 0xc4ceb9fe1a85ec53ull; v ^= v >> 33;
    return (uint32_t)v;
}

// Checks, on n pseudo-random operand pairs, the identities the kernels
// rely on: the folded fixed-point encoding i32(x * (r * 2^k)) equals
// i32((x * r) * 2^k) for 0 <= k <= 60 (x with exponent in [-80, 40], r in
// [2^-30, 2^30]), the reciprocal __frcp_rn(d) equals the IEEE quotient
// 1 / d, and div_by the IEEE quotient, for random dividends, for dividends
// whose quotient lies next to a midpoint of two f32 values, and for the cell
// sizes and volumes of grids of 1 to 4,096 cells; also the f32 -> i32 conversion on NaN, infinities and out-of-range
// values.  counts[0] = identity mismatches, counts[1] = conversion mismatch
// code, counts[2] = the raw hardware conversion of a NaN (informational).
__global__ void k_selftest(uint64_t n, uint64_t seed, unsigned long long* counts) {
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long bad = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t a = mix32(seed ^ (i * 2 + 0)), b = mix32(seed ^ (i * 2 + 1));
        int ex = (int)(a % 121u) - 80, er = (int)((a >> 8) % 61u) - 30, k = (int)((a >> 16) % 61u);
        float x = __uint_as_float((a & 0x80000000u) | ((uint32_t)(ex + 127) << 23) | (b & 0x7fffffu));
        float r = __uint_as_float(((uint32_t)(er + 127) << 23) | ((b >> 9) & 0x7fffffu) | ((a & 1u) << 22));
        if (i & 1) r = -r;
        float p2 = __uint_as_float((uint32_t)(k + 127) << 23);
        float rk = __fmul_rn(r, p2);
        if (f2i(__fmul_rn(__fmul_rn(x, r), p2)) != f2i(__fmul_rn(x, rk))) bad++;
        if (__float_as_uint(__frcp_rn(r)) != __float_as_uint(__fdiv_rn(1.0f, r))) bad++;
        // divisors: |r|, a range over a cell count, the volume of such cells, significands of all ones
        const uint32_t m = (a >> 4) & 3u;
        float d = fabsf(r);
        if (m >= 1u) d = __fdiv_rn((float)(1u + (b & 15u)), (float)(1u + (a >> 20)));
        if (m == 2u) d = __fmul_rn(__fmul_rn(d, d), __fdiv_rn(d, (float)(1u + (b >> 28))));
        if (m == 3u) d = __uint_as_float((__float_as_uint(d) | 0x7fffffu) - (b & 31u));
        const float y = __fdiv_rn(1.0f, d);
        // the dividend nearest to (q + ulp / 2) d, and its neighbours
        const float qm = __uint_as_float(((uint32_t)(127 + (int)(b >> 27)) << 23) | (mix32(seed + i) & 0x7fffffu));
        const double mid = ((double)qm + 0.5 * ((double)__uint_as_float(__float_as_uint(qm) + 1u) - (double)qm)) * (double)d;
        const uint32_t near = __float_as_uint((float)mid);
        for (uint32_t k = 0; k < 4u; k++) {
            const float n = k < 3u ? __uint_as_float(near - 1u + k) : x;
            if (__float_as_uint(div_by(n, d, y)) != __float_as_uint(__fdiv_rn(n, d))) bad++;
        }
    }
    if (bad) atomicAdd(&counts[0], bad);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        volatile float nanv = __int_as_float(0x7fc00000), pinf = __int_as_float(0x7f800000),
                       ninf = __int_as_float(0xff800000), big = 3e9f, nbig = -3e9f, a = 2.9f, b = -2.9f;
        unsigned long long cb = 0;
        if (f2i(nanv) != 0) cb |= 1ull;
        if (f2i(pinf) != 2147483647) cb |= 2ull;
        if (f2i(ninf) != (int)0x80000000) cb |= 4ull;
        if (f2i(big) != 2147483647 || f2i(nbig) != (int)0x80000000) cb |= 8ull;
        if (f2i(b) != -2 || f2i(a) != 2) cb |= 16ull;
        counts[1] = cb;
        counts[2] = (unsigned long long)(uint32_t)__float2int_rz(nanv);
    }
}

// ------------------------------------------------------------------
// launch wrappers
// ------------------------------------------------------------------
template <int E>
int block_size(uint32_t kid) {
    constexpr int W = wide_block<E>();
    switch (kid) {
        case K_P2G_EXPLICIT_128:
        case K_G2P_EXPLICIT_128: return 128;
        case K_PBMPM_ITER_WIDE: if (W) return W; return iter_block<E>();
        case K_PBMPM_FIRST_WIDE:
        case K_FIRST_1F_WIDE:
        case K_FIRST_3F_WIDE: if (W) return W; return first_block<E, 1>();
        case K_FIRST_1F:
        case K_FIRST_3F: return first_block<E, 1>();
        case K_G2P_PBMPM_WIDE:
        case K_G2P_EXPLICIT_WIDE: if (W) return W; return g2p_block<E>();
        case K_P2G_EXPLICIT_WIDE: if (W) return W; return p2g_block<E>();
        case K_PBMPM_ITER: return iter_block<E>();
        case K_P2G_EXPLICIT: return p2g_block<E>();
        case K_G2P_EXPLICIT:
        case K_G2P_PBMPM: return g2p_block<E>();
        default: return kid == K_GRID_DENSE ? 256 : tile_block<E>();   // K_PBMPM_FIRST: its width too
    }
}

template <int E>
size_t smem_bytes(uint32_t kid) {
    constexpr size_t NC = (size_t)(E + 2) * (E + 2) * (E + 2);
    switch (kid) {
        case K_P2G_EXPLICIT:
        case K_G2P_EXPLICIT:
        case K_G2P_PBMPM:
        case K_P2G_EXPLICIT_128:
        case K_G2P_EXPLICIT_128:
        case K_G2P_PBMPM_WIDE:
        case K_P2G_EXPLICIT_WIDE:
        case K_G2P_EXPLICIT_WIDE: return 16 * NC;
        case K_PBMPM_FIRST:
        case K_PBMPM_FIRST_WIDE: return first_smem<E, 0>();
        case K_FIRST_1F:
        case K_FIRST_1F_WIDE: return first_smem<E, 1>();
        case K_FIRST_3F:
        case K_FIRST_3F_WIDE: return first_smem<E, 3>();
        case K_PBMPM_ITER:
        case K_PBMPM_ITER_WIDE: return 32 * NC;
        default: return 0;
    }
}

// every instantiation behind a kernel id (variants share the id's launch shape)
template <int E>
int kernel_ptrs(uint32_t kid, void** out) {
    switch (kid) {
        case K_BIN_INSERT: out[0] = (void*)k_bin_insert<E>; return 1;
        case K_P2G_EXPLICIT: out[0] = (void*)k_p2g_explicit<E, p2g_block<E>()>; return 1;
        case K_G2P_EXPLICIT: out[0] = (void*)k_g2p_integrate<E, false, g2p_block<E>(), 0>; return 1;
        case K_PBMPM_FIRST: out[0] = (void*)k_pbmpm_first<E, first_block<E, 0>(), 0>; return 1;
        case K_FIRST_1F: out[0] = (void*)k_pbmpm_first<E, first_block<E, 1>(), 1>; return 1;
        case K_FIRST_3F: out[0] = (void*)k_pbmpm_first<E, first_block<E, 3>(), 3>; return 1;
        case K_PBMPM_ITER:
            out[0] = (void*)k_pbmpm_iter<E, iter_block<E>(), true>;
            out[1] = (void*)k_pbmpm_iter<E, iter_block<E>(), false>;
            return 2;
        case K_PBMPM_ITER_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_pbmpm_iter<E, wide_block<E>(), true>;
                out[1] = (void*)k_pbmpm_iter<E, wide_block<E>(), false>;
                return 2;
            } else {
                return kernel_ptrs<E>(K_PBMPM_ITER, out);
            }
        case K_PBMPM_FIRST_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_pbmpm_first<E, wide_block<E>(), 0>;
                return 1;
            } else {
                return kernel_ptrs<E>(K_PBMPM_FIRST, out);
            }
        case K_FIRST_1F_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_pbmpm_first<E, wide_block<E>(), 1>;
                return 1;
            } else {
                return kernel_ptrs<E>(K_FIRST_1F, out);
            }
        case K_FIRST_3F_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_pbmpm_first<E, wide_block<E>(), 3>;
                return 1;
            } else {
                return kernel_ptrs<E>(K_FIRST_3F, out);
            }
        case K_G2P_PBMPM_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_g2p_integrate<E, true, wide_block<E>(), 2>;
                out[1] = (void*)k_g2p_integrate<E, true, wide_block<E>(), 0>;
                return 2;
            } else {
                return kernel_ptrs<E>(K_G2P_PBMPM, out);
            }
        case K_P2G_EXPLICIT_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_p2g_explicit<E, wide_block<E>()>;
                return 1;
            } else {
                return kernel_ptrs<E>(K_P2G_EXPLICIT, out);
            }
        case K_G2P_EXPLICIT_WIDE:
            if constexpr (wide_block<E>() != 0) {
                out[0] = (void*)k_g2p_integrate<E, false, wide_block<E>(), 0>;
                return 1;
            } else {
                return kernel_ptrs<E>(K_G2P_EXPLICIT, out);
            }
        case K_G2P_PBMPM:
            out[0] = (void*)k_g2p_integrate<E, true, g2p_block<E>(), 2>;
            out[1] = (void*)k_g2p_integrate<E, true, g2p_block<E>(), 0>;
            return 2;
        case K_GRID_DENSE: out[0] = (void*)k_grid_dense<E>; return 1;
        case K_BIN_PLAN: out[0] = (void*)k_bin_plan<E>; return 1;
        case K_P2G_EXPLICIT_128: out[0] = (void*)k_p2g_explicit<E, 128>; return 1;
        case K_G2P_EXPLICIT_128: out[0] = (void*)k_g2p_integrate<E, false, 128, 0>; return 1;
        default: return 0;
    }
}

template <int E>
cudaError_t configure_tile_kernels(int* blocks_per_sm) {
    for (uint32_t kid : {K_P2G_EXPLICIT, K_G2P_EXPLICIT, K_PBMPM_FIRST, K_PBMPM_ITER, K_G2P_PBMPM, K_GRID_DENSE,
                         K_P2G_EXPLICIT_128, K_G2P_EXPLICIT_128, K_PBMPM_ITER_WIDE, K_PBMPM_FIRST_WIDE,
                         K_G2P_PBMPM_WIDE, K_P2G_EXPLICIT_WIDE, K_G2P_EXPLICIT_WIDE, K_FIRST_1F, K_FIRST_3F,
                         K_FIRST_1F_WIDE, K_FIRST_3F_WIDE}) {
        void* fs[2] = {nullptr, nullptr};
        int nf = kernel_ptrs<E>(kid, fs);
        size_t sm = smem_bytes<E>(kid);
        int nb_min = 1 << 30;
        for (int i = 0; i < nf; i++) {
            cudaError_t e = cudaFuncSetAttribute(fs[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            if (e != cudaSuccess) return e;
            int nb = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fs[i], block_size<E>(kid), sm);
            if (e != cudaSuccess) return e;
            nb_min = nb < nb_min ? nb : nb_min;
        }
        blocks_per_sm[kid] = nb_min > 0 ? nb_min : 1;
    }
    return cudaFuncSetAttribute(k_bin_plan<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_ORDER_SMEM);
}

template <int E>
cudaError_t launch_kernel(uint32_t kid, const Ctx& c, cudaStream_t s, int grid_tiles, uint32_t scene, int apply,
                          int4* out) {
    uint32_t n = c.n_particles;
    uint32_t pblocks = (n + 255u) / 256u;
    switch (kid) {
        case K_CLEAR_TABLE: k_clear_table<<<256, 256, 0, s>>>(c); break;
        case K_BIN_INSERT: if (pblocks) k_bin_insert<E><<<pblocks, 256, 0, s>>>(c); break;
        case K_BIN_PLAN: {
            // neighbour CTAs for the tile storage, at most one per further SM
            uint32_t nb = 0;
            if (c.st_nbr) nb = (uint32_t)std::min<uint64_t>(((uint64_t)c.plan_tiles * 27u + 1023u) / 1024u, 147u);
            const size_t sm = !c.tile_order ? 0 : c.order_bits == 5u ? TILE_ORDER_SMEM : TILE_ORDER_SMEM / 8;
            k_bin_plan<E><<<1u + nb, 1024, sm, s>>>(c);
            break;
        }
        case K_BIN_SCATTER: if (pblocks) k_bin_scatter<<<pblocks, 256, 0, s>>>(c); break;
        case K_P2G_EXPLICIT: k_p2g_explicit<E, p2g_block<E>()><<<grid_tiles, p2g_block<E>(), smem_bytes<E>(kid), s>>>(c); break;
        case K_G2P_EXPLICIT: k_g2p_integrate<E, false, g2p_block<E>(), 0><<<grid_tiles, g2p_block<E>(), smem_bytes<E>(kid), s>>>(c); break;
        case K_PBMPM_FIRST:
        case K_PBMPM_FIRST_WIDE:
        case K_FIRST_1F:
        case K_FIRST_1F_WIDE:
        case K_FIRST_3F:
        case K_FIRST_3F_WIDE: {
            void* f[2] = {nullptr, nullptr};
            kernel_ptrs<E>(kid, f);
            Ctx arg = c;
            void* args[] = {&arg};
            return cudaLaunchKernel(f[0], dim3((unsigned)grid_tiles), dim3((unsigned)block_size<E>(kid)), args,
                                    smem_bytes<E>(kid), s);
        }
        case K_PBMPM_ITER:
            if (c.iter_first) k_pbmpm_iter<E, iter_block<E>(), true><<<grid_tiles, iter_block<E>(), smem_bytes<E>(kid), s>>>(c);
            else k_pbmpm_iter<E, iter_block<E>(), false><<<grid_tiles, iter_block<E>(), smem_bytes<E>(kid), s>>>(c);
            break;
        case K_PBMPM_ITER_WIDE:
            if constexpr (wide_block<E>() != 0) {
                if (c.iter_first) k_pbmpm_iter<E, wide_block<E>(), true><<<grid_tiles, wide_block<E>(), smem_bytes<E>(kid), s>>>(c);
                else k_pbmpm_iter<E, wide_block<E>(), false><<<grid_tiles, wide_block<E>(), smem_bytes<E>(kid), s>>>(c);
            } else {
                return launch_kernel<E>(K_PBMPM_ITER, c, s, grid_tiles, scene, apply, out);
            }
            break;
        case K_G2P_PBMPM_WIDE:
            if constexpr (wide_block<E>() != 0) {
                if (c.g2p_rm) k_g2p_integrate<E, true, wide_block<E>(), 2><<<grid_tiles, wide_block<E>(), smem_bytes<E>(kid), s>>>(c);
                else k_g2p_integrate<E, true, wide_block<E>(), 0><<<grid_tiles, wide_block<E>(), smem_bytes<E>(kid), s>>>(c);
            } else {
                return launch_kernel<E>(K_G2P_PBMPM, c, s, grid_tiles, scene, apply, out);
            }
            break;
        case K_P2G_EXPLICIT_WIDE:
            if constexpr (wide_block<E>() != 0) k_p2g_explicit<E, wide_block<E>()><<<grid_tiles, wide_block<E>(), smem_bytes<E>(kid), s>>>(c);
            else return launch_kernel<E>(K_P2G_EXPLICIT, c, s, grid_tiles, scene, apply, out);
            break;
        case K_G2P_EXPLICIT_WIDE:
            if constexpr (wide_block<E>() != 0) k_g2p_integrate<E, false, wide_block<E>(), 0><<<grid_tiles, wide_block<E>(), smem_bytes<E>(kid), s>>>(c);
            else return launch_kernel<E>(K_G2P_EXPLICIT, c, s, grid_tiles, scene, apply, out);
            break;
        case K_G2P_PBMPM:
            if (c.g2p_rm) k_g2p_integrate<E, true, g2p_block<E>(), 2><<<grid_tiles, g2p_block<E>(), smem_bytes<E>(kid), s>>>(c);
            else k_g2p_integrate<E, true, g2p_block<E>(), 0><<<grid_tiles, g2p_block<E>(), smem_bytes<E>(kid), s>>>(c);
            break;
        case K_COLLIDE: k_collide<<<grid_tiles, 128, 0, s>>>(c); break;
        case K_GRID_DENSE: k_grid_dense<E><<<grid_tiles, 256, 0, s>>>(c, scene, apply, out); break;
        case K_P2G_EXPLICIT_128: k_p2g_explicit<E, 128><<<grid_tiles, 128, smem_bytes<E>(kid), s>>>(c); break;
        case K_G2P_EXPLICIT_128: k_g2p_integrate<E, false, 128, 0><<<grid_tiles, 128, smem_bytes<E>(kid), s>>>(c); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_selftest(uint64_t n, uint64_t seed, unsigned long long* counts, cudaStream_t s) {
    k_selftest<<<1184, 256, 0, s>>>(n, seed, counts);
    return cudaGetLastError();
}

template cudaError_t configure_tile_kernels<4>(int*);
template cudaError_t configure_tile_kernels<8>(int*);
template cudaError_t configure_tile_kernels<12>(int*);
template cudaError_t configure_tile_kernels<14>(int*);
template cudaError_t configure_tile_kernels<16>(int*);
template cudaError_t launch_kernel<4>(uint32_t, const Ctx&, cudaStream_t, int, uint32_t, int, int4*);
template cudaError_t launch_kernel<8>(uint32_t, const Ctx&, cudaStream_t, int, uint32_t, int, int4*);
template cudaError_t launch_kernel<12>(uint32_t, const Ctx&, cudaStream_t, int, uint32_t, int, int4*);
template cudaError_t launch_kernel<14>(uint32_t, const Ctx&, cudaStream_t, int, uint32_t, int, int4*);
template cudaError_t launch_kernel<16>(uint32_t, const Ctx&, cudaStream_t, int, uint32_t, int, int4*);

}  // namespace mpm
