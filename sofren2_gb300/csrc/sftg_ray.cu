/*
 * Ray queries against resident models: sft_raycast_instance (sofren2.c:3733-3837) with
 * sft__intersect_triangle (3705-3731).
 *
 *   model space  sft_m_qinv of the instance transform, applied by sft_m_mul_vec, which uses rows
 *                0-2 only (no translation; the reference's behaviour, kept); the direction is
 *                normalised and the distance limit divided by its inverse length
 *   walk         depth first from a stack, children in slot order: inner children that pass the
 *                slab test are pushed, leaf triangles are tested in place; a hit shortens the
 *                limit, so among equal distances the first triangle found wins, as in the
 *                reference's walk
 *   result       distance back in world scale, position and normal through rows 0-2 of the
 *                transform, the normal normalised (sft_v_norm)
 * Arithmetic is the reference's scalar C sequence in IEEE single precision: the file is built
 * with -fmad=false, and divisions and square roots are the correctly rounded intrinsics.  The walk
 * of many rays holds RAY_STACK entries (an 8-wide BLAS needs 7 per level), that of few whatever the
 * former would stack; a walk that would overflow its stack, or that meets a node or meshlet index
 * outside its model, stops and marks its record with hit = 2.
 */
#include "sftg_types.h"
#include "sftg_kernels.h"
#include "sftg_walk.h"

#define RAY_STACK 128
#define RAY_EPS 1e-6f

struct v3 { float x, y, z; };

__device__ __forceinline__ v3 vsub(v3 a, v3 b) { return { a.x - b.x, a.y - b.y, a.z - b.z }; }
__device__ __forceinline__ float vdot(v3 a, v3 b) { return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z)); }
__device__ __forceinline__ v3 vcross(v3 a, v3 b) {
    return { __fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)), __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
             __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)) };
}
__device__ __forceinline__ v3 vscale(v3 a, float s) { return { __fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s) }; }
__device__ __forceinline__ v3 vnorm(v3 v) {   /* sft_v_norm (1548-1551) */
    const float l = __fsqrt_rn(vdot(v, v));
    return l > RAY_EPS ? vscale(v, __fdiv_rn(1.f, l)) : v3{ 0.f, 0.f, 0.f };
}
/* sft_m_mul_vec (1679-1685): v.x * m[0][j] + v.y * m[1][j] + v.z * m[2][j] */
__device__ __forceinline__ v3 rot3(const float* m, v3 v) {
    return { __fadd_rn(__fadd_rn(__fmul_rn(v.x, m[0]), __fmul_rn(v.y, m[4])), __fmul_rn(v.z, m[8])),
             __fadd_rn(__fadd_rn(__fmul_rn(v.x, m[1]), __fmul_rn(v.y, m[5])), __fmul_rn(v.z, m[9])),
             __fadd_rn(__fadd_rn(__fmul_rn(v.x, m[2]), __fmul_rn(v.y, m[6])), __fmul_rn(v.z, m[10])) };
}
__device__ __forceinline__ float inv_axis(float d) {
    return __fdiv_rn(1.f, fabsf(d) > RAY_EPS ? d : __fmul_rn(RAY_EPS, d < 0.f ? -1.f : 1.f));
}
__device__ __forceinline__ float rmin(float a, float b) { return a < b ? a : b; }   /* SFT_MIN */
__device__ __forceinline__ float rmax(float a, float b) { return a > b ? a : b; }   /* SFT_MAX */

/* The ray in model space. */
struct ray_ms { v3 o, d; float ix, iy, iz, inv_scale; };

__device__ __forceinline__ ray_ms ray_setup(const sftg_ray& R) {
    const float* T = R.transform;
    const float inv[16] = { T[0], T[4], T[8], 0.f, T[1], T[5], T[9], 0.f, T[2], T[6], T[10], 0.f, 0.f, 0.f, 0.f, 1.f };
    ray_ms r;
    r.o = rot3(inv, v3{ R.origin[0], R.origin[1], R.origin[2] });
    r.d = rot3(inv, v3{ R.dir[0], R.dir[1], R.dir[2] });
    r.inv_scale = __fdiv_rn(1.f, __fsqrt_rn(vdot(r.d, r.d)));
    r.d = vscale(r.d, r.inv_scale);
    r.ix = inv_axis(r.d.x); r.iy = inv_axis(r.d.y); r.iz = inv_axis(r.d.z);
    return r;
}

/* slot box against the ray, without the limit */
__device__ __forceinline__ bool slab(const ray_ms& r, float4 mn, float4 mx, float& tmin) {
    const float tx1 = __fmul_rn(__fsub_rn(mn.x, r.o.x), r.ix), tx2 = __fmul_rn(__fsub_rn(mx.x, r.o.x), r.ix);
    const float ty1 = __fmul_rn(__fsub_rn(mn.y, r.o.y), r.iy), ty2 = __fmul_rn(__fsub_rn(mx.y, r.o.y), r.iy);
    const float tz1 = __fmul_rn(__fsub_rn(mn.z, r.o.z), r.iz), tz2 = __fmul_rn(__fsub_rn(mx.z, r.o.z), r.iz);
    tmin = rmax(rmax(rmin(tx1, tx2), rmin(ty1, ty2)), rmin(tz1, tz2));
    const float tmax = rmin(rmin(rmax(tx1, tx2), rmax(ty1, ty2)), rmax(tz1, tz2));
    return (__float_as_uint(mx.w) & 2u) && __float_as_uint(mn.w) != 0xFFFFFFFFu && tmax >= tmin && tmax > 0.f;
}

/* sft__intersect_triangle (3705-3731) */
__device__ __forceinline__ bool triangle(const ray_ms& r, v3 v0, v3 e1, v3 e2, float& t) {
    const v3 p = vcross(r.d, e2);
    const float det = vdot(e1, p);
    if (fabsf(det) < RAY_EPS) return false;
    const float id = __fdiv_rn(1.f, det);
    const v3 tv = vsub(r.o, v0);
    const float u = __fmul_rn(vdot(tv, p), id);
    if (u < 0.f || u > 1.f) return false;
    const v3 qv = vcross(tv, e1);
    const float v = __fmul_rn(vdot(r.d, qv), id);
    if (v < 0.f || __fadd_rn(u, v) > 1.f) return false;
    t = __fmul_rn(vdot(e2, qv), id);
    return t > RAY_EPS;
}

/* the record of a finished walk: the winning triangle tri at t, or none */
__device__ __forceinline__ void store_hit(const sftg_ray& R, bool hit, bool overflow, float t, const sftg_wtri* tri, sftg_ray_hit* out) {
    sftg_ray_hit H;
    H.hit = 0; H.distance = R.max_dist;
    H.pos[0] = H.pos[1] = H.pos[2] = 0.f; H.normal[0] = H.normal[1] = H.normal[2] = 0.f;
    if (hit) {
        const ray_ms r = ray_setup(R);
        float T[16];
#pragma unroll
        for (int q = 0; q < 16; q++) T[q] = R.transform[q];
        const v3 sd = vscale(r.d, t);
        const v3 lh{ __fadd_rn(r.o.x, sd.x), __fadd_rn(r.o.y, sd.y), __fadd_rn(r.o.z, sd.z) };
        const v3 e1{ tri->e1[0], tri->e1[1], tri->e1[2] }, e2{ tri->e2[0], tri->e2[1], tri->e2[2] };
        const v3 ln = vnorm(vcross(e1, e2));   /* sft_v_face_normal */
        const v3 wp = rot3(T, lh), wn = vnorm(rot3(T, ln));
        H.hit = 1; H.distance = __fmul_rn(t, r.inv_scale);
        H.pos[0] = wp.x; H.pos[1] = wp.y; H.pos[2] = wp.z; H.normal[0] = wn.x; H.normal[1] = wn.y; H.normal[2] = wn.z;
    }
    if (overflow) H.hit = 2;
    *out = H;
}

__device__ __forceinline__ bool has_blas(const sftg_ray& R, const sftg_model* models, uint32_t n_models) {
    return R.model >= 0 && (uint32_t)R.model < n_models && models[R.model].blas_count != 0;
}

#define RAY_WARPS 4
#define ALL 0xFFFFFFFFu

/* ---------------------------------------------------------------- many rays
 * 8 lanes per ray, lane c on child slot c of the ray's node.  Walks differ widely in length (on the
 * atrium half take 2 nodes, one in a hundred over 400), so the four groups of a warp step together
 * and each takes the next ray when its own is done: the warp draws 32 rays at a time from a counter
 * and sets them up a lane per ray.  Finished walks leave (triangle, distance) in their hit record;
 * k_ray_records turns those into records, again a thread per ray.
 * Bound by issue (65 % of the slots, 27 of 32 threads) and by the latency of the node loads.  Groups
 * diverging from one another in one warp, with set-up and record by 8 lanes each, ran 9 of 32 threads:
 * 2^20 rays against the atrium took 4.73 ms, now 1.79.  10 and 12 resident CTAs (fewer registers, less L1) took 2.01 and 2.19. */
#define RAY_PENDING 4u   /* of a record's hit word: a walk's result, bit 0 hit, bit 1 overflow */

__global__ void __launch_bounds__(RAY_WARPS * 32)
k_ray_walks(const sftg_ray* __restrict__ rays, uint32_t n, const sftg_model* __restrict__ models, uint32_t n_models,
            const sftg_wslot* __restrict__ wslots, const sftg_wtri* __restrict__ wtris, sftg_ray_hit* __restrict__ hits,
            uint32_t* __restrict__ next)
{
    __shared__ uint32_t s_stack[RAY_WARPS * 4][RAY_STACK];
    __shared__ float s_q[RAY_WARPS][10][32];      /* the warp's drawn rays: origin, direction, inverse direction, limit */
    __shared__ uint32_t s_k[RAY_WARPS][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & 7, first = lane & ~7;
    uint32_t* const stack = s_stack[warp * 4 + (lane >> 3)];
    float (*const q)[32] = s_q[warp];
    int qi = 0, qn = 0;          /* drawn rays taken, held */
    bool dry = false;            /* the counter has passed n */
    int top = 0;
    uint32_t k = ALL;            /* this group's ray */
    ray_ms r;
    float lmax = 0.f, win_t = 0.f;
    uint32_t win = 0, flags = 0, base = 0, count = 0;
    while (true) {
        const bool idle = top == 0;
        if (__any_sync(ALL, idle && (k != ALL || !dry || qi < qn))) {
            if (idle && k != ALL) {
                if (gl == 0) { hits[k].hit = RAY_PENDING | flags; hits[k].distance = win_t; hits[k].pos[0] = __uint_as_float(win); }
                k = ALL;
            }
            if (qi >= qn && !dry) {
                uint32_t k0 = 0;
                if (lane == 0) k0 = atomicAdd(next, 32u);
                k0 = __shfl_sync(ALL, k0, 0);
                dry = k0 >= n;   /* the counter passes n by at most 32 a warp: n is at most SFTG_RAY_MAX */
                const uint32_t mine = k0 + (uint32_t)lane;
                const bool in = !dry && mine < n;
                bool walk = false;
                if (in) {
                    walk = has_blas(rays[mine], models, n_models);
                    if (!walk) store_hit(rays[mine], false, false, 0.f, nullptr, hits + mine);
                }
                const uint32_t m = __ballot_sync(ALL, walk);
                __syncwarp();
                if (walk) {
                    const ray_ms s = ray_setup(rays[mine]);
                    const int at = __popc(m & ((1u << lane) - 1u));
                    q[0][at] = s.o.x; q[1][at] = s.o.y; q[2][at] = s.o.z; q[3][at] = s.d.x; q[4][at] = s.d.y; q[5][at] = s.d.z;
                    q[6][at] = s.ix; q[7][at] = s.iy; q[8][at] = s.iz; q[9][at] = __fdiv_rn(rays[mine].max_dist, s.inv_scale);
                    s_k[warp][at] = mine;
                }
                __syncwarp();
                qi = 0; qn = __popc(m);
            }
            const uint32_t idles = __ballot_sync(ALL, idle);
            const int at = qi + (__popc(idles & ((1u << first) - 1u)) >> 3);
            if (idle && at < qn) {
                k = s_k[warp][at];
                r.o = v3{ q[0][at], q[1][at], q[2][at] }; r.d = v3{ q[3][at], q[4][at], q[5][at] };
                r.ix = q[6][at]; r.iy = q[7][at]; r.iz = q[8][at]; lmax = q[9][at];
                const sftg_model M = models[rays[k].model];
                base = M.blas_base; count = M.blas_count;
                win = 0; win_t = 0.f; flags = 0;
                top = 1;
                if (gl == 0) stack[0] = M.blas_root;
            }
            qi = min(qn, qi + (__popc(idles) >> 3));
            __syncwarp();
            if (!__any_sync(ALL, top > 0)) {
                if (dry && qi >= qn) break;
                continue;
            }
        }
        /* one node per group */
        const bool act = top > 0;
        const uint32_t ni = act ? stack[top - 1] : 0u;
        if (act) top--;
        bool bad = act && ni >= count;
        float4 mn = make_float4(0.f, 0.f, 0.f, 0.f), mx = mn;
        if (act && !bad) {
            const float4* s = (const float4*)(wslots + ((size_t)base + ni) * 8 + gl);
            mn = s[0]; mx = s[1];
        }
        const bool leaf = __float_as_uint(mx.w) & 1u;
        float tmin;
        const bool pass = slab(r, mn, mx, tmin) && act && !bad && tmin < lmax;
        const bool test = pass && leaf;
        if (__any_sync(ALL, test)) {
            bool ok = false;
            float t = 0.f;
            const uint32_t place = ni * 8u + (uint32_t)gl;
            if (test) {
                const float4* w = (const float4*)(wtris + (size_t)base * 8 + place);
                const float4 a = w[0], b = w[1], c = w[2];
                bad = bad || __float_as_uint(c.y) == 0u;
                ok = !bad && triangle(r, v3{ a.x, a.y, a.z }, v3{ a.w, b.x, b.y }, v3{ b.z, b.w, c.x }, t);
            }
            /* slot order against the running limit; a box test that passed with the limit at node entry is
             * re-checked with the current one */
            const uint32_t bads = __ballot_sync(ALL, bad) >> first & 0xFFu, oks = __ballot_sync(ALL, ok) >> first & 0xFFu;
            uint32_t c = bads ? 0u : oks;
            while (__any_sync(ALL, c != 0)) {
                const int s = first + (c ? __ffs(c) - 1 : 0);
                const float tmin_s = __shfl_sync(ALL, tmin, s), t_s = __shfl_sync(ALL, t, s);
                const uint32_t w_s = __shfl_sync(ALL, place, s);
                if (c && tmin_s < lmax && t_s < lmax) { lmax = win_t = t_s; win = w_s; flags |= 1u; }
                c &= c - 1;
            }
        }
        if (__ballot_sync(ALL, bad) >> first & 0xFFu) { flags |= 2u; top = 0; }
        /* the limit does not change while an inner node's children are tested: the passing ones are pushed
         * at once, in slot order */
        const uint32_t pm = __ballot_sync(ALL, pass && !leaf) >> first & 0xFFu;
        if (top + __popc(pm) > RAY_STACK) { flags |= 2u; top = 0; }
        else if (pm) {
            if ((pm >> gl) & 1u) stack[top + __popc(pm & ((1u << gl) - 1u))] = __float_as_uint(mn.w);
            top += __popc(pm);
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(256)
k_ray_records(const sftg_ray* __restrict__ rays, uint32_t n, const sftg_model* __restrict__ models, const sftg_wtri* __restrict__ wtris,
              sftg_ray_hit* __restrict__ hits)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t h = hits[k].hit;
    if (!(h & RAY_PENDING)) return;
    const sftg_wtri* tri = wtris + (size_t)models[rays[k].model].blas_base * 8 + __float_as_uint(hits[k].pos[0]);
    store_hit(rays[k], h & 1u, h & 2u, hits[k].distance, tri, hits + k);
}

/* ---------------------------------------------------------------- few rays
 * A warp per ray; its time is the longest walk's chain of dependent node loads.  Four nodes are
 * expanded per step, the topmost entries of the stack, each replaced in place by its children, or,
 * for a leaf, by the triangles hit: the stack stays in the order of the sequential walk.  A triangle
 * is weighed against the limit when it comes to the top, so the limit is the sequential walk's.  Nodes
 * expanded early may be ones that walk would have skipped; what they hold is rejected by its own
 * box distance, which is no nearer than its ancestors': rounding is monotone and every box lies
 * inside the one its parent holds for it (sftg_model.nested; of every tree built here).  For the same
 * reason an entry whose box lies at or beyond the limit is dropped unread.  A tree a caller gave
 * with other boxes, or with indices outside the model, is walked one node at a time.  600 rays against the atrium (the longest walk 583
 * nodes): 250 us with 8 lanes per ray, one node per step, now 115. */
#define WIDE_STACK 384

struct wide_entry { uint32_t id; float tmin, t; };   /* node, or triangle place | SFTG_WALK_TRI with its distance */

__global__ void __launch_bounds__(RAY_WARPS * 32)
k_ray_wide(const sftg_ray* __restrict__ rays, uint32_t n, const sftg_model* __restrict__ models, uint32_t n_models,
           const sftg_wslot* __restrict__ wslots, const sftg_wtri* __restrict__ wtris, sftg_ray_hit* __restrict__ hits)
{
    __shared__ wide_entry s_stack[RAY_WARPS][WIDE_STACK];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & 7, sub = lane >> 3;
    const uint32_t k = blockIdx.x * RAY_WARPS + (uint32_t)warp;
    if (k >= n) return;
    const sftg_ray& R = rays[k];
    if (!has_blas(R, models, n_models)) {
        if (lane == 0) store_hit(R, false, false, 0.f, nullptr, hits + k);
        return;
    }
    const sftg_model M = models[R.model];
    if (M.blas_root >= M.blas_count) {   /* a caller's; a child outside the tree is found when it is taken */
        if (lane == 0) store_hit(R, false, true, 0.f, nullptr, hits + k);
        return;
    }
    const ray_ms r = ray_setup(R);
    float lmax = __fdiv_rn(R.max_dist, r.inv_scale), win_t = 0.f;
    const sftg_wslot* nodes = wslots + (size_t)M.blas_base * 8;
    const sftg_wtri* tris = wtris + (size_t)M.blas_base * 8;
    wide_entry* const stack = s_stack[warp];
    const bool nested = M.nested != 0;
    const float far = __uint_as_float(0xFF800000u);   /* -inf: an entry never dropped for its box */
    int top = 1;
    if (lane == 0) stack[0] = wide_entry{ M.blas_root, far, 0.f };
    bool overflow = false, hit = false;
    uint32_t win = 0;
    __syncwarp();
    while (top > 0) {
        /* lane l: the l-th entry from the top */
        wide_entry e{ 0u, 0.f, 0.f };
        const bool seen = top - 1 - lane >= 0;
        if (seen) e = stack[top - 1 - lane];
        const bool tri = (e.id & SFTG_WALK_TRI) != 0;
        const bool live = seen && e.tmin < lmax && (!tri || e.t < lmax);
        uint32_t node_m = __ballot_sync(ALL, live && !tri);
        const uint32_t tri_m = __ballot_sync(ALL, live && tri);
        const int first_tri = tri_m ? __ffs(tri_m) - 1 : 32, first_node = node_m ? __ffs(node_m) - 1 : 32;
        if (first_tri < first_node) {   /* triangles above the first node, in order */
            for (uint32_t c = first_node < 32 ? tri_m & ((1u << first_node) - 1u) : tri_m; c; c &= c - 1) {
                const int s = __ffs(c) - 1;
                const float tmin_s = __shfl_sync(ALL, e.tmin, s), t_s = __shfl_sync(ALL, e.t, s);
                const uint32_t id_s = __shfl_sync(ALL, e.id, s);
                if (tmin_s < lmax && t_s < lmax) { lmax = win_t = t_s; win = id_s & ~SFTG_WALK_TRI; hit = true; }
            }
            top = first_node < 32 ? top - first_node : max(0, top - 32);
            __syncwarp();
            continue;
        }
        if (!node_m) { top = max(0, top - 32); __syncwarp(); continue; }
        /* the nodes to expand: up to four, down to the next triangle; one at a time from where the entries left would
         * not hold, after one more step of four (28 entries), what the sequential walk may stack and a leaf's
         * triangles: every walk that fits its RAY_STACK entries fits here */
        if (first_tri < 32) node_m &= (1u << first_tri) - 1u;
        const int most = nested && top <= WIDE_STACK - RAY_STACK - 28 - 8 ? 4 : 1;
        uint32_t pick = node_m;
        for (int g = 0; g < sub; g++) pick &= pick - 1;
        const bool have = pick != 0 && sub < most;
        const int src = have ? __ffs(pick) - 1 : 0;
        const uint32_t ni = __shfl_sync(ALL, e.id, src);
        const int taken = min(most, __popc(node_m));
        const int below = top - 1 - __shfl_sync(ALL, src, (taken - 1) * 8);   /* entries left under the last one taken */
        if (__any_sync(ALL, have && ni >= M.blas_count)) { overflow = true; break; }
        float4 mn = make_float4(0.f, 0.f, 0.f, 0.f), mx = mn;
        if (have) {
            const float4* s = (const float4*)(nodes + (size_t)ni * 8 + gl);
            mn = s[0]; mx = s[1];
        }
        const bool leaf = __float_as_uint(mx.w) & 1u;
        float tmin, t = 0.f;
        bool keep = slab(r, mn, mx, tmin) && have && tmin < lmax, bad = false;
        const uint32_t place = ni * 8u + (uint32_t)gl;
        if (keep && leaf) {
            const float4* w = (const float4*)(tris + place);
            const float4 a = w[0], b = w[1], c = w[2];
            bad = __float_as_uint(c.y) == 0u;
            keep = !bad && triangle(r, v3{ a.x, a.y, a.z }, v3{ a.w, b.x, b.y }, v3{ b.z, b.w, c.x }, t) && t < lmax;
        }
        if (__any_sync(ALL, bad)) { overflow = true; break; }
        /* bottom to top: the last node's outputs first; an inner node's children in slot order (the highest
         * is walked first), a leaf's triangles in reverse (the lowest is weighed first) */
        const uint32_t m = __ballot_sync(ALL, keep);
        const int outs = __popc(m);
        if (below + outs > WIDE_STACK) { overflow = true; break; }
        if (keep) {
            const uint32_t mine = (m >> (sub * 8)) & 0xFFu;
            const int under = sub < 3 ? __popc(m >> (sub * 8 + 8)) : 0;
            const int rank = leaf ? __popc(mine >> (gl + 1)) : __popc(mine & ((1u << gl) - 1u));
            stack[below + under + rank] = leaf ? wide_entry{ SFTG_WALK_TRI | place, tmin, t }
                                               : wide_entry{ __float_as_uint(mn.w), nested ? tmin : far, 0.f };
        }
        top = below + outs;
        __syncwarp();
    }
    if (lane == 0) store_hit(R, hit, overflow, win_t, tris + win, hits + k);
}

#define RAY_GRID (152 * 8)   /* CTAs of the many-ray walk: 8 fit an SM (registers) */
static_assert(RAY_GRID * RAY_WARPS * 32u <= 0xFFFFFFFFu - SFTG_RAY_MAX, "the ray counter does not wrap");

int sftg_launch_raycast(const sftg_ray* rays, uint32_t n, const sftg_model* models, uint32_t n_models, const sftg_wslot* wslots,
                        const sftg_wtri* wtris, uint32_t* next, sftg_ray_hit* hits, cudaStream_t st) {
    if (!n) return 0;
    if (n <= SFTG_RAY_WIDE_MAX) {
        k_ray_wide<<<(n + RAY_WARPS - 1) / RAY_WARPS, RAY_WARPS * 32, 0, st>>>(rays, n, models, n_models, wslots, wtris, hits);
        return 0;
    }
    const cudaError_t e = cudaMemsetAsync(next, 0, 4, st);
    if (e != cudaSuccess) return (int)e;
    const uint32_t want = (n + 32 * RAY_WARPS - 1) / (32 * RAY_WARPS);
    k_ray_walks<<<want < RAY_GRID ? want : RAY_GRID, RAY_WARPS * 32, 0, st>>>(rays, n, models, n_models, wslots, wtris, hits, next);
    k_ray_records<<<(n + 255) / 256, 256, 0, st>>>(rays, n, models, wtris, hits);
    return 0;
}
