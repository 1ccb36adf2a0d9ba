/*
 * Geometry, clipping and binning kernels of the sofren2 render path.
 *
 *   k_geometry  two warps per job of up to 8 meshlets (sft__worker_phase_geom, sofren2.c:4901-5145):
 *               lanes 0-7 run the bounding-sphere frustum test and normal-cone test; each
 *               surviving meshlet is skinned (4 joints), transformed and projected a vertex
 *               per lane, written to the screen-space cache, then its 128 triangles are set
 *               up eight batches at a time (sft__geom_setup_and_bin_batch, 4775-4884): one
 *               8-lane group per batch, shuffles build the batch's tile rectangle and lane mask.
 *   k_clip      near-plane clipping of straddling triangles (4691-4772, 4264-4381); clip
 *               slots come from an exclusive scan of the meshlets' clip counts (or, of few
 *               meshlets, each CTA's own sum), which numbers them in the reference's
 *               single-worker emission order.
 *   k_coarse    one CTA per super-tile (4 x 4 tiles) lists, in slot order, the meshlets of its
 *               view whose tile rectangle overlaps it; run once to count and once to write.
 *   k_bin       one or more CTAs per tile build that tile's payload list in the reference's order
 *               (meshlet, batch, clipped triangles before the batch payload) with ordered
 *               warp-aggregated compaction over the view's meshlets, or its super-tile's
 *               meshlet list (every meshlet that touches the tile is on it, in slot order);
 *               run once to count and once to write.
 *   k_scan_*    a three-phase exclusive scan used for clip slots and tile list offsets.
 */
#include "sftg_types.h"
#include "sftg_lane.cuh"
#include "sftg_kernels.h"

#define GEOM_TEAMS 2    /* meshlet jobs per CTA, two warps each */

/* ----------------------------------------------------------------------------------------- */
/* Two warps per job, a vertex per lane and two rounds of four triangle batches per warp.  Bound by
 * latency: a frame's few hundred to few thousand meshlets leave the SMs a few warps each, and a warp's
 * time is its chain of loads (job, instance, bounds, vertices, indices) and its own instructions.
 * One warp per job (two vertices per lane in turn, bones staged in 16 KB of shared memory per CTA,
 * index bytes loaded where they are used) took, with the clipping after it, 39 us on the skinned 1080p
 * frame (743 meshlets) and 75 on the 1080p 4x atrium, where this takes 27 and 49 (jobs of one meshlet). */
__global__ void __launch_bounds__(GEOM_TEAMS * 64)
k_geometry(const sftg_frame* __restrict__ frames, const sftg_job* __restrict__ jobs, uint32_t n_jobs, float* __restrict__ ss,
           sftg_batch_rec* __restrict__ recs, uint32_t* __restrict__ clip_cnt, uint32_t* __restrict__ clip_tot, int4* __restrict__ mrect)
{
    __shared__ uint4 s_ind[GEOM_TEAMS][32];    /* the meshlet's 512 index bytes */
    __shared__ float s_v[GEOM_TEAMS][3][64];   /* tz sx sy */
    __shared__ int4 s_mr[GEOM_TEAMS];          /* the second warp's share of the meshlet's rectangle */
    __shared__ uint32_t s_clips[GEOM_TEAMS];
    const int team = threadIdx.x >> 6, tt = threadIdx.x & 63, warp = tt >> 5, lane = tt & 31;
    const uint32_t job_i = blockIdx.x * GEOM_TEAMS + team;
    if (job_i >= n_jobs) return;   /* the whole team */
    auto team_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(team + 1) : "memory"); };
    const sftg_job J = jobs[job_i];
    const sftg_frame* F = frames + J.view;
    const sftg_inst* I = &F->inst[J.inst];
    float T[16];
#pragma unroll
    for (int k = 0; k < 16; k++) T[k] = I->T[k];
    const float* bones = (J.skinned && I->bones >= 0) ? F->bones + (size_t)I->bones * 16 : nullptr;

    /* ---- cull (lanes 0..7), 4939-4994 ---- */
    bool inside = false;
    const uint32_t g0 = I->meshlet_base + J.first;
    if (lane < (int)J.count) {
        const float4* cl = (const float4*)(F->ml_cull + (size_t)(g0 + lane) * 8);
        const float4 c0 = cl[0], c1 = cl[1];
        v3 ctr = mk3(c0.x, c0.y, c0.z), ax = mk3(c1.x, c1.y, c1.z);
        if (J.skinned) {
            const int cb = F->ml_info[I->meshlet_base + J.group_first].culling_bone;   /* the group's first bone */
            const float* B = bones + (size_t)cb * 16;
            ctr = xform(ctr, B); ax = xform_dir(ax, B);
        }
        ctr = xform(ctr, T); ax = xform_dir(ax, T);
        const float sxs = fsqrt(T[0] * T[0] + T[1] * T[1] + T[2] * T[2]);
        const float rad = c0.w * sxs;
        ax = vnorm(ax);
        bool in = true;
#pragma unroll
        for (int p = 0; p < 6; p++) {
            const float dist = vdot(ctr, mk3(F->fn[p][0], F->fn[p][1], F->fn[p][2])) + F->fd[p];
            in = in && (dist + rad >= 0.f);
        }
        const v3 vr = sub3(ctr, mk3(F->cam[0], F->cam[1], F->cam[2]));
        const float dd = fsqrt(vdot(vr, vr));
        const float dv = vdot(vr, ax);
        const float thr = fma_(dd, c1.w, rad);
        inside = in && (dv <= thr);
    }
    const uint32_t alive = __ballot_sync(0xFFFFFFFFu, inside) & 0xFFu;   /* the same in both warps */

    const float hw = F->hw, hh = F->hh;
    const float bias_x = hw + F->vpx, scale_y = -hh, bias_y = hh + F->vpy;
    const float* VP = F->vp;
    const int cols = F->cols, rows = F->rows;

    for (uint32_t ln = 0; ln < J.count; ln++) {
        const uint32_t m = J.first + ln;             /* model-relative meshlet index */
        const uint32_t g = I->meshlet_base + m;      /* pool index */
        const uint32_t ssi = F->ss_base + I->ss_offset + m;
        if (!((alive >> ln) & 1u)) {
            /* its records are read only where its rectangle or its clip count says so */
            if (tt == 0) { mrect[ssi] = make_int4(1, 0, 1, 0); clip_tot[ssi] = 0; }
            continue;
        }
        const float* at = F->ml_attr + (size_t)g * 640;
        float* S = ss + (size_t)ssi * SFTG_SS_FLOATS;
        if (warp == 0) s_ind[team][lane] = ((const uint4*)(F->ml_inds + (size_t)g * 512))[lane];
        /* ---- vertex tt (5015-5124) ---- */
        {
            const int v = tt;
            const v3 p = mk3(at[v], at[64 + v], at[128 + v]);
            const v3 n = mk3(at[192 + v], at[256 + v], at[320 + v]);
            const float tu = at[384 + v], tv = at[448 + v], tlu = at[512 + v], tlv = at[576 + v];
            v3 pw, nw;
            if (J.skinned) {
                const int slot = F->ml_info[g].skin_slot;
                const uint16_t* js = F->skin_j + (size_t)slot * 256;
                const uint8_t* ws = F->skin_w + (size_t)slot * 256;
                const float inv255 = 1.f / 255.f;
                v3 vp[4], vn[4]; float wt[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    float M[16];
                    const float4* B = (const float4*)(bones + (size_t)js[k * 64 + v] * 16);
#pragma unroll
                    for (int q = 0; q < 4; q++) { const float4 r = B[q]; M[4 * q] = r.x; M[4 * q + 1] = r.y; M[4 * q + 2] = r.z; M[4 * q + 3] = r.w; }
                    wt[k] = (float)ws[k * 64 + v] * inv255;
                    vp[k] = xform(p, M); vn[k] = xform_dir(n, M);
                }
                pw.x = fma_(vp[0].x, wt[0], fma_(vp[1].x, wt[1], fma_(vp[2].x, wt[2], vp[3].x * wt[3])));
                pw.y = fma_(vp[0].y, wt[0], fma_(vp[1].y, wt[1], fma_(vp[2].y, wt[2], vp[3].y * wt[3])));
                pw.z = fma_(vp[0].z, wt[0], fma_(vp[1].z, wt[1], fma_(vp[2].z, wt[2], vp[3].z * wt[3])));
                nw.x = fma_(vn[0].x, wt[0], fma_(vn[1].x, wt[1], fma_(vn[2].x, wt[2], vn[3].x * wt[3])));
                nw.y = fma_(vn[0].y, wt[0], fma_(vn[1].y, wt[1], fma_(vn[2].y, wt[2], vn[3].y * wt[3])));
                nw.z = fma_(vn[0].z, wt[0], fma_(vn[1].z, wt[1], fma_(vn[2].z, wt[2], vn[3].z * wt[3])));
                pw = xform(pw, T); nw = xform_dir(nw, T);
            } else {
                pw = xform(p, T); nw = xform_dir(n, T);
            }
            const float w = fma_(pw.x, VP[3], fma_(pw.y, VP[7], fma_(pw.z, VP[11], VP[15])));
            const float tx = fma_(pw.x, VP[0], fma_(pw.y, VP[4], fma_(pw.z, VP[8], VP[12])));
            const float ty = fma_(pw.x, VP[1], fma_(pw.y, VP[5], fma_(pw.z, VP[9], VP[13])));
            const float tz = fma_(pw.x, VP[2], fma_(pw.y, VP[6], fma_(pw.z, VP[10], VP[14])));
            const float iw = rcpr(w);
            const float sx = fma_(tx, iw * hw, bias_x), sy = fma_(ty, iw * scale_y, bias_y);
            s_v[team][0][v] = tz; s_v[team][1][v] = sx; s_v[team][2][v] = sy;
            /* vertex-major record (sftg_types.h, SFTG_SS_*): three float4 and one float per vertex */
            ((float4*)(S + SFTG_SS_A))[v] = make_float4(x86nan(sx), x86nan(sy), x86nan(iw), pw.x);
            ((float4*)(S + SFTG_SS_B))[v] = make_float4(pw.y, pw.z, nw.x, nw.y);
            ((float4*)(S + SFTG_SS_C))[v] = make_float4(nw.z, tu, tv, tlu);
            S[SFTG_SS_D + v] = tlv;
        }
        team_sync();
        /* ---- triangle batches: 4 per round, one 8-lane group each, warp w the rounds 2w and 2w + 1 (4775-4884) ---- */
        const uint8_t* ind = (const uint8_t*)s_ind[team];
        const int grp = lane >> 3, tl = lane & 7;
        int4 mr = make_int4(9999, -9999, 9999, -9999);
        uint32_t clips = 0;
#pragma unroll
        for (int round = 0; round < 2; round++) {
            const int b = (warp * 2 + round) * 4 + grp;
            const uint32_t i0 = ind[b * 32 + tl], i1 = ind[b * 32 + 8 + tl], i2 = ind[b * 32 + 16 + tl];
            const bool valid = (int)(i0 | i1 | i2) > 0;
            const float tz0 = s_v[team][0][i0], tz1 = s_v[team][0][i1], tz2 = s_v[team][0][i2];
            const bool ai = (tz0 >= 0.f) && (tz1 >= 0.f) && (tz2 >= 0.f);
            const bool ao = (tz0 < 0.f) && (tz1 < 0.f) && (tz2 < 0.f);
            const bool inter = valid && !(ai || ao);
            uint32_t nclip = inter ? (uint32_t)((tz0 >= 0.f) + (tz1 >= 0.f) + (tz2 >= 0.f)) : 0u;
            const float sx0 = s_v[team][1][i0], sy0 = s_v[team][2][i0];
            const float sx1 = s_v[team][1][i1], sy1 = s_v[team][2][i1];
            const float sx2 = s_v[team][1][i2], sy2 = s_v[team][2][i2];
            const float dx1 = sx1 - sx0, dy1 = sy1 - sy0, dx2 = sx2 - sx0, dy2 = sy2 - sy0;
            const int tx0 = cvtt(vmin(sx0, vmin(sx1, sx2))) >> 6, tx1 = cvtt(vmax(sx0, vmax(sx1, sx2))) >> 6;
            const int ty0 = cvtt(vmin(sy0, vmin(sy1, sy2))) >> 6, ty1 = cvtt(vmax(sy0, vmax(sy1, sy2))) >> 6;
            const bool ok = ai && (fma_(dx1, dy2, -(dy1 * dx2)) > 0.1f) &&
                            tx1 >= 0 && tx0 <= cols - 1 && ty1 >= 0 && ty0 <= rows - 1;
            const uint32_t vm = (__ballot_sync(0xFFFFFFFFu, ok) >> (grp * 8)) & 0xFFu;
            int x0 = ok ? tx0 : 9999, x1 = ok ? tx1 : -9999, y0 = ok ? ty0 : 9999, y1 = ok ? ty1 : -9999;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                x0 = min(x0, __shfl_xor_sync(0xFFFFFFFFu, x0, o));
                x1 = max(x1, __shfl_xor_sync(0xFFFFFFFFu, x1, o));
                y0 = min(y0, __shfl_xor_sync(0xFFFFFFFFu, y0, o));
                y1 = max(y1, __shfl_xor_sync(0xFFFFFFFFu, y1, o));
                nclip += __shfl_xor_sync(0xFFFFFFFFu, nclip, o);
            }
            clips += nclip;
            if (tl == 0) {
                sftg_batch_rec r;
                if (vm) {
                    r.payload = (uint64_t)J.inst | ((uint64_t)m << 24) | ((uint64_t)b << 48) | ((uint64_t)vm << 56);
                    r.x0 = (int16_t)max(-30000, min(30000, x0)); r.x1 = (int16_t)max(-30000, min(30000, x1));
                    r.y0 = (int16_t)max(-30000, min(30000, y0)); r.y1 = (int16_t)max(-30000, min(30000, y1));
                } else { r.payload = 0; r.x0 = 1; r.x1 = 0; r.y0 = 1; r.y1 = 0; }
                recs[(size_t)ssi * 16 + b] = r;
                clip_cnt[(size_t)ssi * 16 + b] = nclip;
            }
            if (vm) { mr.x = min(mr.x, x0); mr.y = max(mr.y, x1); mr.z = min(mr.z, y0); mr.w = max(mr.w, y1); }
        }
        /* meshlet-level rectangle: union of the batch rectangles */
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            mr.x = min(mr.x, __shfl_xor_sync(0xFFFFFFFFu, mr.x, o));
            mr.y = max(mr.y, __shfl_xor_sync(0xFFFFFFFFu, mr.y, o));
            mr.z = min(mr.z, __shfl_xor_sync(0xFFFFFFFFu, mr.z, o));
            mr.w = max(mr.w, __shfl_xor_sync(0xFFFFFFFFu, mr.w, o));
            clips += __shfl_xor_sync(0xFFFFFFFFu, clips, o);
        }
        if (warp == 1 && lane == 0) { s_mr[team] = mr; s_clips[team] = clips; }
        team_sync();   /* also: both warps are done with the vertices and indices */
        if (tt == 0) {
            const int4 o = s_mr[team];
            mrect[ssi] = make_int4(min(mr.x, o.x), max(mr.y, o.y), min(mr.z, o.z), max(mr.w, o.w));
            clip_tot[ssi] = clips + s_clips[team];
        }
    }
}

/* ----------------------------------------------------------------------------------------- */
struct cvert { float tx, ty, tz, w, u, v, lu, lv, px, py, pz, nx, ny, nz; };

SFTG_D cvert lerp_cv(const cvert& a, const cvert& b, float t) {
    cvert r;
    const float* pa = &a.tx; const float* pb = &b.tx; float* pr = &r.tx;
#pragma unroll
    for (int i = 0; i < 14; i++) pr[i] = pa[i] + t * (pb[i] - pa[i]);
    return r;
}

/* the first vertex of a clipped triangle and its edges' cuts, from the vertex's place in the meshlet */
SFTG_D cvert clip_vertex(const float* S, const float* at, uint32_t v, const float* VP) {
    cvert c;
    const float4 sa = ((const float4*)(S + SFTG_SS_A))[v], sb = ((const float4*)(S + SFTG_SS_B))[v];
    const float wx = sa.w, wy = sb.x, wz = sb.y;
    c.w = fma_(wx, VP[3], fma_(wy, VP[7], fma_(wz, VP[11], VP[15])));
    c.tx = fma_(wx, VP[0], fma_(wy, VP[4], fma_(wz, VP[8], VP[12])));
    c.ty = fma_(wx, VP[1], fma_(wy, VP[5], fma_(wz, VP[9], VP[13])));
    c.tz = fma_(wx, VP[2], fma_(wy, VP[6], fma_(wz, VP[10], VP[14])));
    c.u = at[384 + v]; c.v = at[448 + v]; c.lu = at[512 + v]; c.lv = at[576 + v];
    c.px = wx; c.py = wy; c.pz = wz;
    c.nx = sb.z; c.ny = sb.w; c.nz = S[SFTG_SS_C + 4 * v];
    return c;
}

/* one output triangle into its slot, with its tile rectangle; widens mr where it is on screen */
SFTG_D bool clip_store(const sftg_frame* F, uint32_t slot, const cvert& a, const cvert& b, const cvert& c, uint32_t ii, uint32_t m,
                       sftg_clip_tri* clips, int4* clip_rect, int4& mr) {
    if (slot >= F->clip_cap) return false;   /* over capacity: the host grows the pool and re-renders */
    const float hw = F->hw, hh = F->hh;
    sftg_clip_tri ct;
    auto put = [&](int q, const cvert& cv) {
        const float iw = fdiv(1.f, cv.w);
        ct.sx[q] = (cv.tx * iw + 1.f) * hw + F->vpx;
        ct.sy[q] = (-cv.ty * iw + 1.f) * hh + F->vpy;
        ct.iw[q] = iw;
        ct.u[q] = cv.u; ct.v[q] = cv.v; ct.lu[q] = cv.lu; ct.lv[q] = cv.lv;
        ct.px[q] = cv.px; ct.py[q] = cv.py; ct.pz[q] = cv.pz;
        ct.nx[q] = cv.nx; ct.ny[q] = cv.ny; ct.nz[q] = cv.nz;
    };
    put(0, a); put(1, b); put(2, c);
    ct.inst = ii; ct.m = m;
    clips[slot] = ct;
    const float area = (ct.sx[1] - ct.sx[0]) * (ct.sy[2] - ct.sy[0]) - (ct.sy[1] - ct.sy[0]) * (ct.sx[2] - ct.sx[0]);
    int4 rc = make_int4(1, 0, 1, 0);
    bool grew = false;
    if (area > 0.1f) {
        const int x0 = cvtt(floorf(vmin(ct.sx[0], vmin(ct.sx[1], ct.sx[2])))) >> 6;
        const int x1 = cvtt(ceilf(vmax(ct.sx[0], vmax(ct.sx[1], ct.sx[2])))) >> 6;
        const int y0 = cvtt(floorf(vmin(ct.sy[0], vmin(ct.sy[1], ct.sy[2])))) >> 6;
        const int y1 = cvtt(ceilf(vmax(ct.sy[0], vmax(ct.sy[1], ct.sy[2])))) >> 6;
        if (!(x1 < 0 || x0 > F->cols - 1 || y1 < 0 || y0 > F->rows - 1)) {
            rc = make_int4(x0, x1, y0, y1);
            mr.x = min(mr.x, x0); mr.y = max(mr.y, x1); mr.z = min(mr.z, y0); mr.w = max(mr.w, y1);
            grew = true;
        }
    }
    clip_rect[slot] = rc;
    return grew;
}

/* Near-plane clipping (4691-4772, 4264-4349), `per` meshlets per CTA of 16 8-lane groups, one
 * batch of the meshlet per group and one triangle per lane; meshlets that clip nothing cost a look at
 * their count.  Slots follow the meshlet's base (an exclusive scan of the meshlets' counts), then
 * the batches before this one, then the batch's earlier triangles: the reference's order.  Bound by
 * latency: 32 records per warp, four batches at a time, with the vertices in an array indexed by
 * which of them are in front (local memory) took 24 us on the skinned 1080p frame; four meshlets per
 * CTA there leave most of the GPU idle while two or three of one CTA clip in turn. */
#define CLIP_THREADS 128
__global__ void __launch_bounds__(CLIP_THREADS)
k_clip(const sftg_frame* __restrict__ frames, uint32_t n_views, const float* __restrict__ ss,
       const uint32_t* __restrict__ clip_cnt, const uint32_t* __restrict__ clip_tot, uint32_t* clip_base,
       sftg_clip_tri* __restrict__ clips, int4* __restrict__ clip_rect, int4* __restrict__ mrect, uint32_t n_meshlets, uint32_t per,
       uint32_t* __restrict__ total)
{
    const int tid = threadIdx.x, lane = tid & 31, tl = lane & 7, gshift = lane & ~7, b = tid >> 3;
    const uint32_t gmask = 0xFFu << gshift;
    const uint32_t m0 = blockIdx.x * per;
    uint32_t base0 = 0;
    if (total) {   /* one meshlet per CTA: its base is the sum of the counts before it */
        __shared__ uint32_t s_sum[CLIP_THREADS / 32];
        uint32_t sum = 0;
#pragma unroll 4
        for (uint32_t i = tid; i < m0; i += CLIP_THREADS) sum += clip_tot[i];
        sum = __reduce_add_sync(0xFFFFFFFFu, sum);
        if (lane == 0) s_sum[tid >> 5] = sum;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < CLIP_THREADS / 32; w++) base0 += s_sum[w];
        if (tid == 0) {
            clip_base[m0] = base0;
            if (m0 + 1u == n_meshlets) *total = base0 + clip_tot[m0];
        }
    }
    const uint32_t mine = m0 + (uint32_t)lane;
    uint32_t pending = __ballot_sync(0xFFFFFFFFu, lane < (int)per && mine < n_meshlets && clip_tot[mine] != 0);
    for (; pending; pending &= pending - 1) {
        const uint32_t ssi = m0 + (uint32_t)(__ffs(pending) - 1);
        /* the batch's outputs and those of the batches before it */
        const uint32_t cnt = clip_cnt[(size_t)ssi * 16 + (lane & 15)];
        uint32_t before = cnt;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, before, o, 16);
            if ((lane & 15) >= o) before += t;
        }
        before -= cnt;
        const uint32_t have = __shfl_sync(0xFFFFFFFFu, cnt, b), first = __shfl_sync(0xFFFFFFFFu, before, b);
        if (!have) continue;   /* whole group */
        /* the view, then the instance, owning this screen-space slot (both laid out in order) */
        uint32_t v = 0;
        for (uint32_t k = 0; k < n_views; k++) if (frames[k].ss_base <= ssi && frames[k].total_ss) v = k;
        const sftg_frame* F = frames + v;
        const uint32_t lss = ssi - F->ss_base;
        uint32_t ii = 0;
        for (uint32_t k = 0; k < F->n_inst; k++) if (F->inst[k].ss_offset <= lss) ii = k;
        const sftg_inst* I = &F->inst[ii];
        const uint32_t m = lss - I->ss_offset, g = I->meshlet_base + m;
        const float* at = F->ml_attr + (size_t)g * 640;
        const float* S = ss + (size_t)ssi * SFTG_SS_FLOATS;
        const uint8_t* ind = F->ml_inds + (size_t)g * 512;
        const float* VP = F->vp;
        const uint32_t q0 = ind[b * 32 + tl], q1 = ind[b * 32 + 8 + tl], q2 = ind[b * 32 + 16 + tl];
        int nc = 0;
        cvert v0, v1, v2;      /* one in front: that vertex, the next, the one before; two: the one behind, the one before, the next */
        if ((int)(q0 | q1 | q2) > 0) {
            auto depth = [&](uint32_t q) {
                const float4 sa = ((const float4*)(S + SFTG_SS_A))[q], sb = ((const float4*)(S + SFTG_SS_B))[q];
                return fma_(sa.w, VP[2], fma_(sb.x, VP[6], fma_(sb.y, VP[10], VP[14])));
            };
            const float d0 = depth(q0), d1 = depth(q1), d2 = depth(q2);
            const bool f0 = d0 >= 0.f, f1 = d1 >= 0.f, f2 = d2 >= 0.f;
            const bool ai = f0 && f1 && f2, ao = (d0 < 0.f) && (d1 < 0.f) && (d2 < 0.f);
            if (!(ai || ao)) {
                /* sft__clip_triangle_near_plane (4264-4349) */
                const int mask = (int)f0 | ((int)f1 << 1) | ((int)f2 << 2);
                const bool one = mask == 1 || mask == 2 || mask == 4;
                const int p = one ? mask >> 1 : (~mask & 7) >> 1;                 /* the pivot's place */
                const uint32_t qp = p == 0 ? q0 : (p == 1 ? q1 : q2);
                const uint32_t qn = p == 0 ? q1 : (p == 1 ? q2 : q0), qb = p == 0 ? q2 : (p == 1 ? q0 : q1);   /* next, before */
                v0 = clip_vertex(S, at, qp, VP);
                v1 = clip_vertex(S, at, one ? qn : qb, VP);
                v2 = clip_vertex(S, at, one ? qb : qn, VP);
                nc = one ? 1 : 2;
            }
        }
        /* exclusive scan of the output counts over the group's 8 triangles */
        int incl = nc;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int t = __shfl_up_sync(gmask, incl, o, 8);
            if (tl >= o) incl += t;
        }
        const uint32_t slot = (total ? base0 : clip_base[ssi]) + first + (uint32_t)(incl - nc);
        int4 mr = make_int4(0x7FFFFFFF, (int)0x80000000, 0x7FFFFFFF, (int)0x80000000);
        bool grew = false;
        if (nc == 1) {
            const float tab = fdiv(v0.tz, v0.tz - v1.tz), tac = fdiv(v0.tz, v0.tz - v2.tz);
            grew = clip_store(F, slot, v0, lerp_cv(v0, v1, tab), lerp_cv(v0, v2, tac), ii, m, clips, clip_rect, mr);
        } else if (nc == 2) {
            const float tab = fdiv(v1.tz, v1.tz - v0.tz), tcb = fdiv(v2.tz, v2.tz - v0.tz);
            const cvert nab = lerp_cv(v1, v0, tab), ncb = lerp_cv(v2, v0, tcb);
            const bool g0 = clip_store(F, slot, v1, nab, v2, ii, m, clips, clip_rect, mr);
            const bool g1 = clip_store(F, slot + 1, nab, ncb, v2, ii, m, clips, clip_rect, mr);
            grew = g0 || g1;
        }
        /* several triangles and batches of one meshlet may clip: widen its rectangle atomically
         * (min / max commute, so the result does not depend on the order) */
        if (grew) {
            atomicMin(&mrect[ssi].x, mr.x); atomicMax(&mrect[ssi].y, mr.y);
            atomicMin(&mrect[ssi].z, mr.z); atomicMax(&mrect[ssi].w, mr.w);
        }
    }
}

/* ----------------------------------------------------------------------------------------- */
#define BIN_THREADS 256

SFTG_D bool rect_has(int x0, int x1, int y0, int y1, int tx, int ty) { return x0 <= tx && tx <= x1 && y0 <= ty && ty <= y1; }

/* Payloads of a meshlet per half warp (lane & 15 = batch) that land on tile (tx, ty), counted or written
 * in reference order: for each batch, its clipped triangles (slot order) then its batch payload.
 * Returns the meshlet's total on the half's lanes; `on` is false for a half without a meshlet. */
SFTG_D uint32_t bin_meshlet(const sftg_batch_rec* recs, const uint32_t* clip_cnt, const uint32_t* clip_tot, const uint32_t* clip_base,
                            const int4* clip_rect, uint32_t clip_cap, uint32_t vclip, bool on, uint32_t ssi, int tx, int ty, int lane,
                            uint64_t* out)
{
    const int b = lane & 15;
    uint32_t cnt = 0, nclip = 0, cb = 0;
    sftg_batch_rec r; r.payload = 0; r.x0 = 1; r.x1 = 0; r.y0 = 1; r.y1 = 0;
    uint32_t clipping = 0;
    if (on) { r = recs[(size_t)ssi * 16 + b]; clipping = clip_tot[ssi]; }
    if (__any_sync(0xFFFFFFFFu, clipping != 0)) {
        if (clipping) { nclip = clip_cnt[(size_t)ssi * 16 + b]; cb = clip_base[ssi]; }
        uint32_t incl = nclip;   /* the meshlet's clip slots, batch after batch */
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o, 16);
            if (b >= o) incl += v;
        }
        cb += incl - nclip;
        for (uint32_t k = 0; k < nclip && cb + k < clip_cap; k++) {
            const int4 q = clip_rect[cb + k];
            cnt += rect_has(q.x, q.y, q.z, q.w, tx, ty);
        }
    }
    const bool whole = r.payload != 0 && rect_has(r.x0, r.x1, r.y0, r.y1, tx, ty);
    cnt += whole;
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o, 16);
        if (b >= o) incl += v;
    }
    if (out && cnt) {
        uint64_t* o = out + (incl - cnt);
        for (uint32_t k = 0; k < nclip && cb + k < clip_cap; k++) {
            const int4 q = clip_rect[cb + k];
            if (rect_has(q.x, q.y, q.z, q.w, tx, ty)) *o++ = (uint64_t)(cb + k - vclip);
        }
        if (whole) *o = r.payload;
    }
    return __shfl_sync(0xFFFFFFFFu, incl, lane | 15);
}

#define COARSE_THREADS 1024   /* a super-tile scans its view's meshlet slots 1024 at a time */

__global__ void __launch_bounds__(COARSE_THREADS)
k_coarse(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ stile_view, const int4* __restrict__ mrect,
         uint32_t* __restrict__ stile_count, const uint32_t* __restrict__ stile_start, uint32_t* __restrict__ stile_list)
{
    __shared__ uint32_t s_wsum[COARSE_THREADS / 32];
    const int gst = blockIdx.x;                         /* batch-wide super-tile index */
    const sftg_frame* F = frames + stile_view[gst];
    const int st = gst - (int)F->stile_base;
    const int sx0 = (st % (int)F->scols) * SFTG_STILE, sy0 = (st / (int)F->scols) * SFTG_STILE;
    const int sx1 = sx0 + SFTG_STILE - 1, sy1 = sy0 + SFTG_STILE - 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t* out = nullptr;
    if (stile_list) {
        /* over capacity: the host grows the lists and re-renders; write nothing */
        if ((uint64_t)stile_start[gst] + stile_count[gst] > F->stile_cap) return;
        out = stile_list + stile_start[gst];
    }
    uint32_t running = 0;
    for (uint32_t base = 0; base < F->total_ss; base += COARSE_THREADS) {
        const uint32_t s = F->ss_base + base + tid;
        bool hit = false;
        if (base + tid < F->total_ss) {
            const int4 q = mrect[s];   /* inclusive tile rectangle x0, x1, y0, y1; empty when x0 > x1 */
            hit = q.x <= q.y && q.z <= q.w && q.x <= sx1 && q.y >= sx0 && q.z <= sy1 && q.w >= sy0;
        }
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, hit);
        if (lane == 0) s_wsum[warp] = __popc(bal);
        __syncthreads();
        uint32_t off = 0, tot = 0;
        for (int w = 0; w < COARSE_THREADS / 32; w++) { if (w < warp) off += s_wsum[w]; tot += s_wsum[w]; }
        if (out && hit) out[running + off + __popc(bal & ((1u << lane) - 1u))] = s;
        running += tot;
        __syncthreads();
    }
    if (!stile_list && tid == 0) stile_count[gst] = running;
}

/* One CTA per (tile, segment): the payloads of the segment's share of the tile's candidate meshlets
 * (all of the view's slots, or its super-tile's list), BIN_CHUNK candidates at a time.  Run once to
 * count (tile_pay null), once to write.  Bound by latency: with a CTA per tile the few tiles of a small
 * frame scanned thousands of meshlets one after the other (155x106 over the atrium 0.44 ms for both
 * passes), and above 1024 slots the super-tile lists, made first, cost three launches, 33 us; now
 * frames of under 1024 tiles cut the candidates over up to 608 CTAs instead. */
#define BIN_CHUNK (4 * BIN_THREADS)
__global__ void __launch_bounds__(BIN_THREADS)
k_bin(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ tile_view, uint32_t nseg, const sftg_batch_rec* __restrict__ recs,
      const uint32_t* __restrict__ clip_cnt, const uint32_t* __restrict__ clip_tot, const uint32_t* __restrict__ clip_base,
      const int4* __restrict__ clip_rect, const int4* __restrict__ mrect, const uint32_t* __restrict__ stile_count,
      const uint32_t* __restrict__ stile_start, const uint32_t* __restrict__ stile_list, uint32_t* __restrict__ seg_count,
      const uint32_t* __restrict__ seg_start, const uint32_t* __restrict__ tile_count, uint64_t* __restrict__ tile_pay,
      const uint32_t* __restrict__ total, float2* __restrict__ vis, uint32_t* __restrict__ raster_done)
{
    __shared__ uint32_t s_hits[BIN_CHUNK];
    __shared__ uint32_t s_cnt[BIN_CHUNK];
    __shared__ uint32_t s_wsum[4][BIN_THREADS / 32];
    __shared__ uint32_t s_total;
    const int gtile = (int)(blockIdx.x / nseg);         /* batch-wide tile index */
    const uint32_t seg = blockIdx.x - (uint32_t)gtile * nseg;
    const sftg_frame* F = frames + tile_view[gtile];
    const int tile = gtile - (int)F->tile_base;
    const int tx = tile % F->cols, ty = tile / F->cols;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = lane >> 4;
    const uint32_t n_ss = F->total_ss;
    /* clipped payloads carry the view's own slot numbers (slots restart at 0 per frame) */
    const uint32_t vclip = n_ss ? clip_base[F->ss_base] : 0u;
    uint64_t* out = nullptr;
    if (tile_pay) {
        if (sftg_raster_parts(tile_count[gtile], *total, F->samples) > 1u) {   /* rastered in parts, merged into a cleared buffer */
            const int n = F->samples * SFTG_TILE_PX / 2;
            float4* v = (float4*)(vis + F->vis_base + (size_t)tile * F->samples * SFTG_TILE_PX);
            for (int i = (int)seg * BIN_THREADS + tid; i < n; i += (int)nseg * BIN_THREADS) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (seg == 0 && tid < 4) raster_done[gtile * 4 + tid] = 0u;
        }
        /* over capacity: the host grows the buffer and re-renders; write nothing */
        if ((uint64_t)seg_start[blockIdx.x] + seg_count[blockIdx.x] > F->tile_cap) return;
        if (seg_count[blockIdx.x] == 0) return;
        out = tile_pay + seg_start[blockIdx.x];
    }
    /* the meshlets that can touch this tile: its super-tile's list, in slot order, or every slot
     * of the view when the view has no coarse lists (scols == 0) */
    uint32_t n_cand = n_ss;
    const uint32_t* cand = nullptr;
    if (F->scols) {
        const uint32_t gst = F->stile_base + (uint32_t)((ty / SFTG_STILE) * (int)F->scols + tx / SFTG_STILE);
        n_cand = stile_count[gst];
        if ((uint64_t)stile_start[gst] + n_cand > F->stile_cap) n_cand = 0;   /* lists overflowed: the host re-renders */
        cand = stile_list + stile_start[gst];
    }
    const uint32_t share = (n_cand + nseg - 1) / nseg, c0 = min(n_cand, seg * share), c1 = min(n_cand, c0 + share);
    uint32_t running = 0;
    for (uint32_t base = c0; base < c1; base += BIN_CHUNK) {
        /* four candidates per thread, their loads in flight together; candidate order is (j, tid) */
        uint32_t s[4], bal[4];
        bool hit[4], any = false;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t i = base + (uint32_t)(j * BIN_THREADS + tid);
            hit[j] = false; s[j] = 0;
            if (i < c1) {
                s[j] = cand ? cand[i] : F->ss_base + i;
                const int4 q = mrect[s[j]];
                hit[j] = rect_has(q.x, q.y, q.z, q.w, tx, ty);
            }
            any = any || hit[j];
        }
        if (!__syncthreads_or(any)) continue;   /* no meshlet of this chunk touches the tile */
        /* ordered compaction of hit meshlets */
#pragma unroll
        for (int j = 0; j < 4; j++) {
            bal[j] = __ballot_sync(0xFFFFFFFFu, hit[j]);
            if (lane == 0) s_wsum[j][warp] = __popc(bal[j]);
        }
        __syncthreads();
        uint32_t nh = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t off = nh;
            for (int w = 0; w < BIN_THREADS / 32; w++) { if (w < warp) off += s_wsum[j][w]; nh += s_wsum[j][w]; }
            if (hit[j]) s_hits[off + __popc(bal[j] & ((1u << lane) - 1u))] = s[j];
        }
        __syncthreads();
        /* per-hit payload counts, two meshlets per warp at a time */
        for (uint32_t h0 = warp * 2; h0 < nh; h0 += BIN_THREADS / 16) {
            const uint32_t h = h0 + half;
            const uint32_t c = bin_meshlet(recs, clip_cnt, clip_tot, clip_base, clip_rect, F->clip_cap, vclip, h < nh, h < nh ? s_hits[h] : 0u,
                                           tx, ty, lane, nullptr);
            if ((lane & 15) == 0 && h < nh) s_cnt[h] = c;
        }
        __syncthreads();
        if (out) {
            if (warp == 0) {   /* exclusive scan of the hit counts, 32 per lane; total in s_total */
                const uint32_t per = (nh + 31) / 32;
                uint32_t local = 0;
                for (uint32_t k = 0; k < per; k++) { const uint32_t h = (uint32_t)lane * per + k; local += h < nh ? s_cnt[h] : 0u; }
                uint32_t incl = local;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o); if (lane >= o) incl += t; }
                uint32_t acc = incl - local;
                for (uint32_t k = 0; k < per; k++) {
                    const uint32_t h = (uint32_t)lane * per + k;
                    if (h < nh) { const uint32_t c = s_cnt[h]; s_cnt[h] = acc; acc += c; }
                }
                if (lane == 31) s_total = incl;
            }
            __syncthreads();
            for (uint32_t h0 = warp * 2; h0 < nh; h0 += BIN_THREADS / 16) {   /* ordered writes */
                const uint32_t h = h0 + half;
                bin_meshlet(recs, clip_cnt, clip_tot, clip_base, clip_rect, F->clip_cap, vclip, h < nh, h < nh ? s_hits[h] : 0u, tx, ty, lane,
                            out + running + (h < nh ? s_cnt[h] : 0u));
            }
            running += s_total;
        } else {
            uint32_t mine = 0;
            for (uint32_t h = tid; h < nh; h += BIN_THREADS) mine += s_cnt[h];
            running += mine;   /* this thread's share, summed at the end */
        }
        __syncthreads();
    }
    if (!out && !tile_pay) {
        const uint32_t w = __reduce_add_sync(0xFFFFFFFFu, running);
        if (lane == 0) s_wsum[0][warp] = w;
        __syncthreads();
        if (tid == 0) {
            uint32_t all = 0;
            for (int k = 0; k < BIN_THREADS / 32; k++) all += s_wsum[0][k];
            seg_count[blockIdx.x] = all;
        }
    }
}

/* ----------------------------------------------------------------------------------------- */
/* three-phase exclusive scan of u32 (n <= 1024 * 1024 * 4) */
#define SCAN_BLOCK 1024

SFTG_D uint32_t block_excl_scan(uint32_t v, uint32_t* s_w, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o); if (lane >= o) incl += t; }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t x = lane < nw ? s_w[lane] : 0, xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, xi, o); if (lane >= o) xi += t; }
        if (lane < nw) s_w[lane] = xi - x;
        if (lane == 31) s_w[32] = xi;
    }
    __syncthreads();
    const uint32_t r = s_w[warp] + incl - v;
    if (total) *total = s_w[32];
    __syncthreads();
    return r;
}

__global__ void k_scan_reduce(const uint32_t* __restrict__ in, uint32_t n, uint32_t* __restrict__ sums) {
    __shared__ uint32_t s_w[33];
    uint32_t acc = 0;
    const uint32_t base = blockIdx.x * SCAN_BLOCK * 4;
    for (int k = 0; k < 4; k++) { const uint32_t i = base + k * SCAN_BLOCK + threadIdx.x; if (i < n) acc += in[i]; }
    uint32_t tot;
    block_excl_scan(acc, s_w, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void k_scan_top(uint32_t* __restrict__ sums, uint32_t nb, uint32_t* __restrict__ total_out) {
    __shared__ uint32_t s_w[33];
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nb; base += SCAN_BLOCK) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < nb ? sums[i] : 0;
        uint32_t tot;
        const uint32_t e = block_excl_scan(v, s_w, &tot);
        if (i < nb) sums[i] = e + carry;
        carry += tot;
    }
    if (threadIdx.x == 0 && total_out) *total_out = carry;
}

/* the whole scan in one CTA for small inputs (n <= SFTG_SCAN_SMALL): each thread a run of
 * consecutive elements, one block scan of the run sums */
__global__ void __launch_bounds__(SCAN_BLOCK)
k_scan_small(const uint32_t* __restrict__ in, uint32_t n, uint32_t* __restrict__ out, uint32_t* __restrict__ total_out) {
    __shared__ uint32_t s_w[33];
    const uint32_t per = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
    const uint32_t i0 = threadIdx.x * per;
    uint32_t acc = 0;
    for (uint32_t k = 0; k < per; k++) { const uint32_t i = i0 + k; if (i < n) acc += in[i]; }
    uint32_t tot;
    uint32_t e = block_excl_scan(acc, s_w, &tot);
    for (uint32_t k = 0; k < per; k++) { const uint32_t i = i0 + k; if (i < n) { const uint32_t x = in[i]; out[i] = e; e += x; } }
    if (threadIdx.x == 0 && total_out) *total_out = tot;
}

__global__ void k_scan_down(const uint32_t* __restrict__ in, uint32_t n, const uint32_t* __restrict__ sums, uint32_t* __restrict__ out) {
    __shared__ uint32_t s_w[33];
    const uint32_t base = blockIdx.x * SCAN_BLOCK * 4;
    const uint32_t i0 = base + threadIdx.x * 4;
    uint32_t v[4], acc = 0;
    for (int k = 0; k < 4; k++) { const uint32_t i = i0 + k; v[k] = i < n ? in[i] : 0; acc += v[k]; }
    uint32_t e = block_excl_scan(acc, s_w, nullptr) + sums[blockIdx.x];
    for (int k = 0; k < 4; k++) { const uint32_t i = i0 + k; if (i < n) out[i] = e; e += v[k]; }
}
