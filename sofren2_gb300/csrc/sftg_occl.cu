/*
 * The per-frame proxy occlusion pass (inside sft_present, sofren2.c:8163-8280):
 *   k_occl_tlas        one warp per packet (light, batch of 8 proxies, one of 3 disk rays): ray
 *                      set-up and packet frustum, a lane per proxy, corner and plane, and the TLAS
 *                      walk; each reached static instance becomes a (packet, instance) pair
 *   k_occl_blas_expand one warp per pair: a small BLAS to the bottom, the top levels of a large one,
 *                      whose deeper nodes become items
 *   k_occl_blas_walk   one warp per item
 *   k_occl_finalize    light_vis = 3 - blocked rays per (proxy, light)
 * The reference traces each packet serially and stops once every ray is blocked; the OR of
 * hits it accumulates does not depend on the visiting order, so splitting the walk across
 * warps, and taking four stacked nodes per step, gives the same light_vis.  Stacks are fixed-size in
 * shared memory; an overflow sets a status bit instead of writing out of bounds.
 * Bound by the chain of dependent node loads.
 */
#include "sftg_types.h"
#include "sftg_lane.cuh"
#include "sftg_kernels.h"

#define OCC_WARPS 4
/* entries; one node a step from half on, so trees of up to 14 levels fit whatever is hit (7 entries a level) */
#define OCC_STACK 256         /* TLAS */
#define OCC_WALK_STACK 256    /* BLAS */
#define OCC_ALL 0xFFFFFFFFu

/* a box against six planes (normal, distance) in shared memory (sft__frustum_vs_bvh_node, 3906-3968) */
SFTG_D bool box_inside(float mnx, float mny, float mnz, float mxx, float mxy, float mxz, const float4* f) {
    const float cx = (mxx + mnx) * 0.5f, cy = (mxy + mny) * 0.5f, cz = (mxz + mnz) * 0.5f;
    const float ex = (mxx - mnx) * 0.5f, ey = (mxy - mny) * 0.5f, ez = (mxz - mnz) * 0.5f;
    bool in = true;
#pragma unroll
    for (int p = 0; p < 6; p++) {
        const float4 q = f[p];
        const float r = fma_(fabsf(q.x), ex, fma_(fabsf(q.y), ey, fabsf(q.z) * ez));
        const float dc = fma_(q.x, cx, fma_(q.y, cy, q.z * cz));
        const float dist = dc + q.w;
        in = in && (dist + r >= 0.f);
    }
    return in;
}

/* sft_m_view_look_at (1737-1770) */
SFTG_D void view_look_at(v3 pos, v3 target, v3 up, float* m) {
    const v3 fwd = snorm(sub3(target, pos));
    if (fabsf(fwd.x) < 1e-6f && fabsf(fwd.z) < 1e-6f) up = mk3(0.f, 0.f, -1.f);
    up = snorm(sub3(up, scl3(fwd, sdot(up, fwd))));
    const v3 right = cross3(up, fwd);
    m[0] = right.x; m[1] = up.x; m[2] = fwd.x; m[3] = 0.f;
    m[4] = right.y; m[5] = up.y; m[6] = fwd.y; m[7] = 0.f;
    m[8] = right.z; m[9] = up.z; m[10] = fwd.z; m[11] = 0.f;
    m[12] = -sdot(pos, right); m[13] = -sdot(pos, up); m[14] = -sdot(pos, fwd); m[15] = 1.f;
}

/* status bits */
#define OCC_STACK_OVERFLOW 1u     /* also: a node index outside its tree */
#define OCC_UNDEFINED_FRUSTUM 2u
#define OCC_PAIR_OVERFLOW 4u

/* one traced packet: 8 rays from proxy points toward one point of the light disk */
struct __align__(16) sftg_packet {
    float4 f[6];                /* world-space packet frustum: normal, distance */
    float o[3][8], e[3][8];     /* ray origins and ends (origin + L) */
    uint32_t active;
    uint32_t hits;              /* OR of the rays found blocked */
    uint32_t pad[2];
};

SFTG_D float min8(float v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = fminf(v, __shfl_xor_sync(OCC_ALL, v, o));
    return v;
}
SFTG_D float max8(float v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = fmaxf(v, __shfl_xor_sync(OCC_ALL, v, o));
    return v;
}

/* sft__build_packet_frustum (3970-4084) for the packet whose ray k starts at (x, y, z) on lane k of
 * every 8; lane p < 6 of each warp gets plane p.  Returns false when the reference leaves the side
 * planes undefined (a cluster corner at or behind the light); those planes then never cull. */
SFTG_D bool packet_frustum(float x, float y, float z, uint32_t active, v3 lpos, float lrad, int lane, float4& plane) {
    const int k = lane & 7;
    const bool on = (active >> k) & 1u;
    const float mnx = min8(on ? fminf(x, 1e9f) : 1e9f), mny = min8(on ? fminf(y, 1e9f) : 1e9f), mnz = min8(on ? fminf(z, 1e9f) : 1e9f);
    const float mxx = max8(on ? fmaxf(x, -1e9f) : -1e9f), mxy = max8(on ? fmaxf(y, -1e9f) : -1e9f), mxz = max8(on ? fmaxf(z, -1e9f) : -1e9f);
    v3 ctr = mk3(0.f, 0.f, 0.f); int nv = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {   /* in ray order */
        const float sx = __shfl_sync(OCC_ALL, x, i), sy = __shfl_sync(OCC_ALL, y, i), sz = __shfl_sync(OCC_ALL, z, i);
        if ((active >> i) & 1u) { ctr.x = ctr.x + sx; ctr.y = ctr.y + sy; ctr.z = ctr.z + sz; nv++; }
    }
    ctr.x = fdiv(ctr.x, (float)nv); ctr.y = fdiv(ctr.y, (float)nv); ctr.z = fdiv(ctr.z, (float)nv);
    const v3 lf0 = snorm(sub3(ctr, lpos));
    v3 up = mk3(0.f, 1.f, 0.f);
    if (fabsf(lf0.y) > 0.99f) up = mk3(1.f, 0.f, 0.f);
    float lv[16];
    view_look_at(lpos, ctr, up, lv);
    /* corner k of the cluster's box in light space */
    const float bx = (k & 1) ? mxx : mnx, by = (k & 2) ? mxy : mny, bz = (k & 4) ? mxz : mnz;
    const float cxv = bx * lv[0] + by * lv[4] + bz * lv[8] + 1.f * lv[12];
    const float cyv = bx * lv[1] + by * lv[5] + bz * lv[9] + 1.f * lv[13];
    const float czv = bx * lv[2] + by * lv[6] + bz * lv[10] + 1.f * lv[14];
    const bool invalid = __any_sync(OCC_ALL, czv < 1e-6f);
    const float qx = fdiv(cxv, czv), qy = fdiv(cyv, czv);
    const float mnxz = min8(fminf(qx, 1e9f)), mxxz = max8(fmaxf(qx, -1e9f)), mnyz = min8(fminf(qy, 1e9f)), mxyz = max8(fmaxf(qy, -1e9f));
    const v3 lr = mk3(lv[0], lv[4], lv[8]), lu = mk3(lv[1], lv[5], lv[9]), lf = mk3(lv[2], lv[6], lv[10]);
    v3 n;
    if (k < 4) {
        v3 nl = mk3(1.f, 0.f, -mnxz);
        if (k == 1) nl = mk3(-1.f, 0.f, mxxz);
        if (k == 2) nl = mk3(0.f, 1.f, -mnyz);
        if (k == 3) nl = mk3(0.f, -1.f, mxyz);
        const v3 q = snorm(nl);
        n = add3(scl3(lr, q.x), add3(scl3(lu, q.y), scl3(lf, q.z)));
    } else {
        n = k == 4 ? lf : mk3(-lf.x, -lf.y, -lf.z);
    }
    plane = make_float4(n.x, n.y, n.z, -sdot(n, lpos) + (k == 5 ? lrad : 0.1f));
    if (k < 4 && invalid) plane = make_float4(0.f, 0.f, 0.f, 1e30f);
    return !invalid;
}

/* Phase A: one warp per packet (light, proxy batch, ray): ray set-up, packet frustum and the
 * TLAS walk (sofren2.c:8178-8269, 4086-4135); every static instance the frustum reaches becomes
 * a (packet, instance) pair for phase B.  Bound by the chain of loads and the pair counter's atomic per
 * step: with one node per step the phase took 48 us on a 160x90 thumbnail and 54 on the static 640x360
 * scene, now 43 and 45; 94 and 89 on the mixed materials 1333x717. */
__global__ void __launch_bounds__(OCC_WARPS * 32)
k_occl_tlas(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ packet_view, uint32_t n_packets,
            sftg_packet* __restrict__ packets, uint2* __restrict__ pairs, uint32_t* __restrict__ n_pairs, uint32_t max_pairs,
            uint32_t* __restrict__ status)
{
    __shared__ uint32_t s_stack[OCC_WARPS][OCC_STACK];
    __shared__ float4 s_f[OCC_WARPS][6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = lane & 7;
    const uint32_t pk = blockIdx.x * OCC_WARPS + warp;   /* batch-wide packet index */
    if (pk >= n_packets) return;
    const sftg_frame* F = frames + packet_view[pk];
    const uint32_t lpk = pk - F->packet_base;            /* packet index within the view */
    const uint32_t pc = F->n_proxies, nbatch = (pc + 7) / 8;
    const uint32_t ray = lpk % 3, b = (lpk / 3) % nbatch, l = lpk / (3 * nbatch), pb = b * 8;
    const sftg_point_light L = F->point[l];
    const v3 lpos = mk3(L.pos[0], L.pos[1], L.pos[2]);
    /* lane k: proxy pb + k */
    const bool on = pb + k < pc;
    sftg_proxy px;
    px.posa[0] = px.posa[1] = px.posa[2] = px.posb[0] = px.posb[1] = px.posb[2] = 0.f;
    if (on) px = F->proxies[pb + k];
    const uint32_t am = __ballot_sync(OCC_ALL, on) & 0xFFu;
    /* batch centre, summed in proxy order, and light-disk targets, identical on every lane */
    const v3 cen = mk3((px.posa[0] + px.posb[0]) * 0.5f, (px.posa[1] + px.posb[1]) * 0.5f, (px.posa[2] + px.posb[2]) * 0.5f);
    v3 bc = mk3(0.f, 0.f, 0.f); int na = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const float sx = __shfl_sync(OCC_ALL, cen.x, q), sy = __shfl_sync(OCC_ALL, cen.y, q), sz = __shfl_sync(OCC_ALL, cen.z, q);
        if ((am >> q) & 1u) { bc.x = bc.x + sx; bc.y = bc.y + sy; bc.z = bc.z + sz; na++; }
    }
    if (na > 0) bc = scl3(bc, fdiv(1.f, (float)na));
    const v3 ldir = snorm(sub3(lpos, bc));
    float mnv = fabsf(ldir.x); v3 card = mk3(1.f, 0.f, 0.f);
    if (fabsf(ldir.y) < mnv) { mnv = fabsf(ldir.y); card = mk3(0.f, 1.f, 0.f); }
    if (fabsf(ldir.z) < mnv) card = mk3(0.f, 0.f, 1.f);
    const v3 perp = mk3(ldir.y * card.z - ldir.z * card.y, ldir.z * card.x - ldir.x * card.z, ldir.x * card.y - ldir.y * card.x);
    const v3 lright = snorm(perp);
    const v3 lup = cross3(lright, ldir);
    const float r = 0.1f;
    v3 tg;
    if (ray == 0) tg = add3(lpos, scl3(lup, r));
    else if (ray == 1) tg = add3(lpos, add3(scl3(lright, r * 0.866025f), scl3(lup, -r * 0.5f)));
    else tg = add3(lpos, add3(scl3(lright, -r * 0.866025f), scl3(lup, -r * 0.5f)));
    float x = 0.f, y = 0.f, z = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
    if (on) {
        if (ray == 0) { x = px.posa[0]; y = px.posa[1]; z = px.posa[2]; }
        else if (ray == 1) { x = px.posb[0]; y = px.posb[1]; z = px.posb[2]; }
        else { x = cen.x; y = cen.y; z = cen.z; }
        lx = tg.x - x; ly = tg.y - y; lz = tg.z - z;
    }
    sftg_packet* P = &packets[pk];
    if (lane < 8) {
        P->o[0][k] = x; P->o[1][k] = y; P->o[2][k] = z;
        P->e[0][k] = x + lx; P->e[1][k] = y + ly; P->e[2][k] = z + lz;
    }
    if (lane == 0) { P->active = am; P->hits = 0; }
    if (am == 0) return;
    float4 plane;
    if (!packet_frustum(x, y, z, am, lpos, L.radius, lane, plane) && lane == 0) atomicOr(status, OCC_UNDEFINED_FRUSTUM);
    if (lane < 6) { P->f[lane] = plane; s_f[warp][lane] = plane; }
    if (F->tlas_count == 0) return;
    if (F->tlas_root >= F->tlas_count) {   /* children are checked where they are pushed */
        if (lane == 0) atomicOr(status, OCC_STACK_OVERFLOW);
        return;
    }
    int top = 1;
    if (lane == 0) s_stack[warp][0] = F->tlas_root;
    __syncwarp();
    /* four nodes per step, lane (node kq, child k): pushes (inner nodes) and pair emission (leaves)
     * are warp-aggregated; the pairs' order does not matter (hits are OR-ed) */
    const int kq = lane >> 3;
    while (top > 0) {
        const int take = top <= OCC_STACK / 2 ? min(top, 4) : 1;   /* which bounds the stack by 7 entries a level */
        const bool have = kq < take;
        const uint32_t ni = have ? s_stack[warp][top - 1 - kq] : 0u;
        top -= take;
        __syncwarp();
        const sftg_bvh_node* nd = &F->tlas[ni];
        uint32_t ch = SFTG_INVALID;
        bool mine = false, leaf = false;
        if (have) {
            ch = nd->child[k]; leaf = nd->leaf != 0;
            mine = ch != SFTG_INVALID && box_inside(nd->mn[0][k], nd->mn[1][k], nd->mn[2][k], nd->mx[0][k], nd->mx[1][k], nd->mx[2][k], s_f[warp]);
        }
        const uint32_t pm = __ballot_sync(OCC_ALL, mine && !leaf);
        if (pm) {
            if (__ballot_sync(OCC_ALL, mine && !leaf && ch >= F->tlas_count) || top + __popc(pm) > OCC_STACK) {
                if (lane == 0) atomicOr(status, OCC_STACK_OVERFLOW);
                return;
            }
            if (mine && !leaf) s_stack[warp][top + __popc(pm & ((1u << lane) - 1u))] = ch;
            top += __popc(pm);
        }
        bool emit = false;
        const uint32_t ii = ch & ~0x80000000u;
        if (mine && leaf && ii < F->n_inst) {
            const sftg_model* Md = &F->models[F->inst[ii].model];
            emit = !(Md->bone_count > 0 || Md->blas_count == 0);   /* static instances only */
        }
        const uint32_t em = __ballot_sync(OCC_ALL, emit);
        if (em) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(n_pairs, (uint32_t)__popc(em));
            base = __shfl_sync(OCC_ALL, base, 0);
            if (emit) {
                const uint32_t slot = base + __popc(em & ((1u << lane) - 1u));
                if (slot < max_pairs) pairs[slot] = make_uint2(pk, ii);
                else atomicOr(status, OCC_PAIR_OVERFLOW);
            }
        }
        __syncwarp();   /* the pushes, before they are popped */
    }
}

/* Phase B: a warp per (packet, static instance) pair, in two launches.  The packet frustum and
 * rays are taken into model space, then the BLAS is walked four nodes per step, one child AABB per
 * lane (4137-4238); leaf triangles are taken four at a time, lanes (triangle k of 4, ray r of 8)
 * running the any-hit test (3840-3904).  Hits are OR-ed into the packet, which is what the reference
 * accumulates in any visiting order, so a walk can be split into independent sub-walks: the expand
 * launch walks a small BLAS to the bottom; of a larger one the top two or three levels, and turns each
 * deeper node that passes the frustum test into an item (pair, node), which the walk launch runs to
 * the bottom: the phase takes as long as its longest sub-walk.  Both start from the rays the packet already
 * has blocked, which only skips tests whose outcome is already recorded.
 * Occlusion phase with one node per step, 8 of 32 lanes on it, and the triangle's indices and
 * vertices read one after the other: atrium 1080p 4x 0.444 ms, 1279x719 1x 0.218, skinned 1080p 2x
 * 0.145, 48 views 4.25; now 0.120, 0.093, 0.036 and 0.87.  Items at depth 2 only: 0.137, 0.100, 0.050,
 * 0.87; at depth 3 for the batch too 1.04; at depth 3 for small trees too, the 600-node spheres of the static scene, of four levels, are walked by one warp
 * each (0.214 against 0.054). */
#define OCC_WHOLE 64u     /* nodes of a BLAS walked to the bottom by the expand launch */
#define OCC_SHALLOW 1024u /* nodes up to which the nodes at depth 2 become items, else those at depth 3 */
#define OCC_DEEP 2048u    /* packets up to which that is so: more of them fill the GPU with items of depth 2 */
#define OCC_GRID_CTAS (152 * 8)

struct occ_walk {
    v3 lo, ld;      /* ray lane & 7 in model space */
    float tmax;
    uint32_t full;
};

/* The packet's 8 rays in model space, shared by the warp, for the ray-box prune below. */
struct occ_rays { float ox[8], oy[8], oz[8], ix[8], iy[8], iz[8], tmax[8]; };

/* Optional second cull (sftg_tuning.occl_ray_prune) of a child the frustum test kept: it survives if
 * one of the rays still unblocked passes through its box grown by a margin.  A well-conditioned
 * any-hit test only reports triangles within rounding of the ray, so the result is unchanged; but
 * when a ray grazes a triangle's plane (|a| just above the test's 1e-6 threshold while its true value
 * is rounding noise) the reference's u, v and t are noise and it can report a hit far from the ray,
 * which this cull would skip.  That is why it is off by default. */
SFTG_D bool ray_box_hit(float4 mn, float4 mx, const occ_rays& R, uint32_t open_rays) {
    const float lo[3] = { mn.x, mn.y, mn.z }, hi[3] = { mx.x, mx.y, mx.z };
    float blo[3], bhi[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float m = 1e-4f * (fabsf(lo[a]) + fabsf(hi[a]) + (hi[a] - lo[a])) + 1e-5f;
        blo[a] = lo[a] - m; bhi[a] = hi[a] + m;
    }
    bool hit = false;
    for (int r = 0; r < 8; r++) {
        if (!((open_rays >> r) & 1u)) continue;
        const float o[3] = { R.ox[r], R.oy[r], R.oz[r] }, id[3] = { R.ix[r], R.iy[r], R.iz[r] };
        float tn = -3.0e38f, tf = 3.0e38f;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float t1 = (blo[a] - o[a]) * id[a], t2 = (bhi[a] - o[a]) * id[a];
            tn = fmaxf(tn, fminf(t1, t2)); tf = fminf(tf, fmaxf(t1, t2));
        }
        const float tm = R.tmax[r] * 1.0001f + 1e-4f;
        hit = hit || (tn <= tf && tf >= -1e-4f && tn <= tm);
    }
    return hit;
}

/* lanes 0..7 publish their ray; inverse directions with zero components made huge, not infinite */
SFTG_D void occ_rays_publish(const occ_walk& w, occ_rays& R, int lane) {
    if (lane < 8) {
        R.ox[lane] = w.lo.x; R.oy[lane] = w.lo.y; R.oz[lane] = w.lo.z;
        R.ix[lane] = w.ld.x != 0.f ? 1.f / w.ld.x : copysignf(1e30f, w.ld.x);
        R.iy[lane] = w.ld.y != 0.f ? 1.f / w.ld.y : copysignf(1e30f, w.ld.y);
        R.iz[lane] = w.ld.z != 0.f ? 1.f / w.ld.z : copysignf(1e30f, w.ld.z);
        R.tmax[lane] = w.tmax;
    }
}

/* the packet in the instance's model space: lane p < 6 its plane p (into f), lane r & 7 its ray r */
SFTG_D void occ_pair_setup(const sftg_inst* I, const sftg_packet* P, int lane, occ_walk& w, float4* f) {
    const float* M = I->T;
    __syncwarp();   /* the warp's previous walk is done with f */
    if (lane < 6) {
        const float4 pf = P->f[lane];
        const float nx = pf.x, ny = pf.y, nz = pf.z, d = pf.w;
        const float nmx = nx * M[0] + ny * M[1] + nz * M[2];
        const float nmy = nx * M[4] + ny * M[5] + nz * M[6];
        const float nmz = nx * M[8] + ny * M[9] + nz * M[10];
        const float dot_t = nx * M[12] + ny * M[13] + nz * M[14];
        const float dm = dot_t + d;
        const float il = fdiv(1.f, fsqrt(nmx * nmx + nmy * nmy + nmz * nmz));
        f[lane] = make_float4(nmx * il, nmy * il, nmz * il, dm * il);
    }
    /* sft_m_qinv (1693-1712) */
    float im[16];
    im[0] = M[0]; im[1] = M[4]; im[2] = M[8]; im[3] = 0.f;
    im[4] = M[1]; im[5] = M[5]; im[6] = M[9]; im[7] = 0.f;
    im[8] = M[2]; im[9] = M[6]; im[10] = M[10]; im[11] = 0.f;
    for (int a = 0; a < 3; a++) im[12 + a] = -(M[12] * im[a] + M[13] * im[4 + a] + M[14] * im[8 + a]);
    im[15] = 1.f;
    const int r = lane & 7;
    w.lo = xform(mk3(P->o[0][r], P->o[1][r], P->o[2][r]), im);
    const v3 le = xform(mk3(P->e[0][r], P->e[1][r], P->e[2][r]), im);
    const v3 Lv = sub3(le, w.lo);
    w.tmax = fsqrt(vdot(Lv, Lv));
    w.ld = vnorm_fast(Lv);
    w.full = P->active;
}

/* Walks the BLAS of model Md from `start`.  With EXPAND and `split` > 0, a child that would sit at depth
 * `split` is handed out as an item instead of being pushed (or pushed after all when the
 * item list is full).  Returns the rays found blocked. */
template <bool EXPAND>
SFTG_D uint32_t occ_walk_from(const sftg_frame* F, const sftg_model& Md, const occ_walk& w, const float4* f, uint32_t sat,
                              uint32_t start, uint32_t split, uint32_t pair, uint32_t* stack, occ_rays& R, bool prune, uint2* items,
                              uint32_t* n_items, uint32_t max_items, uint32_t* status, int lane) {
    const int r = lane & 7, kq = lane >> 3;   /* child or ray, node or triangle */
    const uint32_t full = w.full;
    int top = 1;
    if (lane == 0) stack[0] = start;      /* entry: node | depth << 29 (depth only tracked when expanding) */
    if (prune) occ_rays_publish(w, R, lane);
    __syncwarp();
    const sftg_wslot* slots = F->wslots + (size_t)Md.blas_base * 8;
    const sftg_wtri* tris = F->wtris + (size_t)Md.blas_base * 8;
    uint32_t guard = 0;
    while (top > 0 && sat != full) {
        /* the four topmost nodes; one where the stack is half full, which bounds it by 7 entries a level */
        const int take = top <= OCC_WALK_STACK / 2 ? min(top, 4) : 1;
        const bool have = kq < take;
        const uint32_t ent = have ? stack[top - 1 - kq] : 0u;
        top -= take;
        __syncwarp();
        const uint32_t ni = ent & 0x1FFFFFFFu, depth = ent >> 29;
        float4 mn = make_float4(0.f, 0.f, 0.f, 0.f), mx = mn;
        if (have) {
            const float4* sl = (const float4*)(slots + (size_t)ni * 8 + r);
            mn = sl[0]; mx = sl[1];
        }
        const uint32_t ch = __float_as_uint(mn.w);
        const bool leaf = __float_as_uint(mx.w) & 1u;
        bool in = have && ch != SFTG_INVALID && box_inside(mn.x, mn.y, mn.z, mx.x, mx.y, mx.z, f);
        if (prune && in) in = ray_box_hit(mn, mx, R, full & ~sat);
        /* inner nodes' children: one ballot for the checks, one atomic for the items, one stack write per lane */
        const bool mine = in && !leaf;
        const uint32_t tm = __ballot_sync(OCC_ALL, mine);
        if (tm) {
            guard += (uint32_t)__popc(tm);
            if (__ballot_sync(OCC_ALL, mine && (ch >= Md.blas_count || ch >= (1u << 29))) || guard > (1u << 24)) {
                if (lane == 0) atomicOr(status, OCC_STACK_OVERFLOW);
                return sat;
            }
            uint32_t pm = tm;
            if (EXPAND) {
                const bool hand = mine && split && depth + 1 >= split;
                const uint32_t hm = __ballot_sync(OCC_ALL, hand);
                if (hm) {
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(n_items, (uint32_t)__popc(hm));
                    base = __shfl_sync(OCC_ALL, base, 0) + __popc(hm & ((1u << lane) - 1u));
                    const bool placed = hand && base < max_items;
                    if (placed) items[base] = make_uint2(pair, ch);
                    pm = tm & ~__ballot_sync(OCC_ALL, placed);   /* children without an item slot are walked here */
                }
            }
            if (top + __popc(pm) > OCC_WALK_STACK) {
                if (lane == 0) atomicOr(status, OCC_STACK_OVERFLOW);
                return sat;
            }
            if ((pm >> lane) & 1u) stack[top + __popc(pm & ((1u << lane) - 1u))] = ch | (EXPAND ? min(depth + 1u, 7u) << 29 : 0u);
            top += __popc(pm);
        }
        /* leaves: the triangles whose boxes are inside, four at a time, lane = (triangle kq, ray r) */
        uint32_t m = __ballot_sync(OCC_ALL, in && leaf);
        while (m && sat != full) {
            uint32_t mm = m;
            for (int q = 0; q < kq; q++) mm &= mm - 1;
            const int src = mm ? __ffs(mm) - 1 : 0;
            const bool test = mm != 0 && ((full & ~sat) >> r & 1u);
            const uint32_t nt = __shfl_sync(OCC_ALL, ni, src);
            for (int q = 0; q < 4; q++) m &= m - 1;
            bool hit = false;
            if (test) {
                const float4* tq = (const float4*)(tris + (size_t)nt * 8 + (src & 7));
                const float4 ta = tq[0], tb = tq[1], tc = tq[2];
                const v3 v0 = mk3(ta.x, ta.y, ta.z), e1 = mk3(ta.w, tb.x, tb.y), e2 = mk3(tb.z, tb.w, tc.x);
                const v3 h = cross3(w.ld, e2);
                const float a = vdot(e1, h);
                hit = __float_as_uint(tc.y) != 0u && fabsf(a) > 1e-6f;
                const float fr = rcpr(a);
                const v3 sv = sub3(w.lo, v0);
                const float u = fr * vdot(sv, h);
                hit = hit && u >= 0.f && u <= 1.f;
                const v3 q = cross3(sv, e1);
                const float v = fr * vdot(w.ld, q);
                hit = hit && v >= 0.f && (u + v) <= 1.f;
                const float tt = fr * vdot(e2, q);
                hit = hit && tt > 1e-6f && tt < w.tmax;
            }
            const uint32_t bal = __ballot_sync(OCC_ALL, hit);
            sat |= (bal | (bal >> 8) | (bal >> 16) | (bal >> 24)) & 0xFFu;
        }
        __syncwarp();
    }
    return sat;
}

SFTG_D uint32_t occ_hits_now(const sftg_packet* P) { return *(volatile const uint32_t*)&P->hits; }

__global__ void __launch_bounds__(OCC_WARPS * 32)
k_occl_blas_expand(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ packet_view, sftg_packet* __restrict__ packets,
                   const uint2* __restrict__ pairs, const uint32_t* __restrict__ n_pairs, uint32_t max_pairs,
                   uint2* __restrict__ items, uint32_t* __restrict__ n_items, uint32_t max_items, uint32_t* __restrict__ status,
                   int prune, uint32_t deep)
{
    __shared__ uint32_t s_stack[OCC_WARPS][OCC_WALK_STACK];
    __shared__ float4 s_f[OCC_WARPS][6];
    __shared__ occ_rays s_rays[OCC_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t np = min(*n_pairs, max_pairs);
    for (uint32_t item = blockIdx.x * OCC_WARPS + warp; item < np; item += gridDim.x * OCC_WARPS) {
        const uint2 pr = pairs[item];
        const sftg_frame* F = frames + packet_view[pr.x];
        sftg_packet* P = &packets[pr.x];
        const uint32_t known = occ_hits_now(P) & P->active;
        if (known == P->active) continue;            /* every ray already blocked */
        const sftg_inst* I = &F->inst[pr.y];
        const sftg_model Md = F->models[I->model];
        if (Md.blas_root >= Md.blas_count) {   /* a caller's tree */
            if (lane == 0) atomicOr(status, OCC_STACK_OVERFLOW);
            continue;
        }
        occ_walk w;
        occ_pair_setup(I, P, lane, w, s_f[warp]);
        const uint32_t sat = occ_walk_from<true>(F, Md, w, s_f[warp], known, Md.blas_root,
                                                 Md.blas_count <= OCC_WHOLE ? 0u : (Md.blas_count <= OCC_SHALLOW ? 2u : deep), item, s_stack[warp],
                                                 s_rays[warp], prune != 0, items, n_items, max_items, status, lane);
        if (lane == 0 && (sat & ~known)) atomicOr(&P->hits, sat);
        __syncwarp();
    }
}

__global__ void __launch_bounds__(OCC_WARPS * 32)
k_occl_blas_walk(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ packet_view, sftg_packet* __restrict__ packets,
                 const uint2* __restrict__ pairs, const uint2* __restrict__ items, const uint32_t* __restrict__ n_items,
                 uint32_t max_items, uint32_t* __restrict__ status, int prune)
{
    __shared__ uint32_t s_stack[OCC_WARPS][OCC_WALK_STACK];
    __shared__ float4 s_f[OCC_WARPS][6];
    __shared__ occ_rays s_rays[OCC_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t ni = min(*n_items, max_items);
    for (uint32_t it = blockIdx.x * OCC_WARPS + warp; it < ni; it += gridDim.x * OCC_WARPS) {
        const uint2 itm = items[it];
        const uint2 pr = pairs[itm.x];
        const sftg_frame* F = frames + packet_view[pr.x];
        sftg_packet* P = &packets[pr.x];
        const uint32_t known = occ_hits_now(P) & P->active;
        if (known == P->active) continue;            /* every ray already blocked */
        const sftg_inst* I = &F->inst[pr.y];
        const sftg_model Md = F->models[I->model];
        occ_walk w;
        occ_pair_setup(I, P, lane, w, s_f[warp]);
        const uint32_t sat = occ_walk_from<false>(F, Md, w, s_f[warp], known, itm.y, 0u, 0, s_stack[warp], s_rays[warp], prune != 0,
                                                  nullptr, nullptr, 0, status, lane);
        if (lane == 0 && (sat & ~known)) atomicOr(&P->hits, sat);
        __syncwarp();
    }
}

/* Phase C: light_vis[p][l] = 3 - rays blocked (8169-8276), 0 past the view's lights and where it
 * traces no packets; one thread per (batch-wide proxy, light column). */
__global__ void k_occl_finalize(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ prox_view, uint32_t n_proxies,
                                const sftg_packet* __restrict__ packets, uint8_t* __restrict__ light_vis)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_proxies * 64) return;
    const uint32_t gp = i >> 6, l = i & 63;
    const sftg_frame* F = frames + prox_view[gp];
    const uint32_t pc = F->n_proxies, lc = min(F->n_point, 64u), nbatch = (pc + 7) / 8;
    uint8_t seen = 0;
    if (l < lc && F->n_packets) {
        const uint32_t p = gp - F->prox_base, b = p / 8, k = p % 8;
        const sftg_packet* P = packets + F->packet_base;
        int blocked = 0;
        for (int ray = 0; ray < 3; ray++) blocked += (P[(l * nbatch + b) * 3 + ray].hits >> k) & 1u;
        seen = (uint8_t)(3 - blocked);
    }
    light_vis[(size_t)gp * 64 + l] = seen;
}

size_t sftg_packet_bytes() { return sizeof(sftg_packet); }

void sftg_launch_occlusion(const sftg_frame* frames, const uint16_t* packet_view, uint32_t n_packets, const uint16_t* prox_view,
                           uint32_t n_proxies, uint32_t max_inst, void* packets, uint2* pairs, uint32_t* n_pairs,
                           uint32_t max_pairs, uint32_t items_per_pair, uint8_t* light_vis, uint32_t* status, int ray_prune,
                           cudaStream_t st) {
    if (n_proxies && !n_packets) k_occl_finalize<<<(n_proxies * 64 + 255) / 256, 256, 0, st>>>(frames, prox_view, n_proxies, (const sftg_packet*)packets, light_vis);
    if (!n_packets) return;
    k_occl_tlas<<<(n_packets + OCC_WARPS - 1) / OCC_WARPS, OCC_WARPS * 32, 0, st>>>(frames, packet_view, n_packets,
                                                                                   (sftg_packet*)packets, pairs, n_pairs, max_pairs, status);
    /* the item list shares the pair buffer's tail: pairs take [0, max_pairs), items the rest */
    uint2* items = pairs + max_pairs;
    uint32_t* n_items = n_pairs + 1;
    const uint32_t max_items = max_pairs * items_per_pair;
    const uint64_t want = (uint64_t)n_packets * (max_inst ? max_inst : 1);
    const uint32_t mp = want < max_pairs ? (uint32_t)want : max_pairs;
    const uint32_t g1 = (mp + OCC_WARPS - 1) / OCC_WARPS;
    k_occl_blas_expand<<<g1 < OCC_GRID_CTAS ? g1 : OCC_GRID_CTAS, OCC_WARPS * 32, 0, st>>>(frames, packet_view, (sftg_packet*)packets,
                                                                                         pairs, n_pairs, max_pairs, items, n_items,
                                                                                         max_items, status, ray_prune,
                                                                                         n_packets <= OCC_DEEP ? 3u : 2u);
    k_occl_blas_walk<<<OCC_GRID_CTAS, OCC_WARPS * 32, 0, st>>>(frames, packet_view, (sftg_packet*)packets, pairs, items, n_items,
                                                               max_items, status, ray_prune);
    k_occl_finalize<<<(n_proxies * 64 + 255) / 256, 256, 0, st>>>(frames, prox_view, n_proxies, (const sftg_packet*)packets, light_vis);
}
