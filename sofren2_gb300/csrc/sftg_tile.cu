/*
 * Per-tile raster and resolve (sft__worker_phase_rasterize, sofren2.c:6756-6813,
 * sft__rast_simd_batch 5148-5499, sft__resolve_tile 5809-6753).
 *
 * k_raster: a CTA per work item, a part of a 64x64 tile's payload list on the tile or a band of its
 * rows (sftg_raster_parts; a band keeps the triangles that reach it, whose rows it walks from the
 * triangle's first row exactly as the whole tile's walk would).  The reference walks the tile's list in order and keeps a
 * sample when z > stored z (strict), so a sample ends holding the largest z, and among equal z
 * the earliest triangle.  That final state does not depend on the order triangles are visited,
 * so each sample is a 64-bit shared-memory word (z bits << 32 | ~order) updated with atomicMax,
 * where order = list position * 8 + lane; only z > 0 ever wins (the buffer starts at 0).
 * Coverage and z are replayed bit-exactly: a group of 8 * S threads takes one triangle's rows, a thread
 * one sample of a pixel column of every aligned 8-pixel chunk (tri_raster), with the reference's
 * trivial-accept / AA guard-band choices; the AA chunk skip is a group vote.  The decoded visibility buffer
 * (depth, vid) goes to global memory, where it stays L2-resident, with the tile's depth range.
 *
 * k_resolve: 1 to 16 CTAs per tile (sftg_resolve_split), each a share of its 4x2 blocks (the
 * reference's AVX2 lanes).  A warp lists the covered (pixel, triangle) fragments of 4 to 16
 * neighbouring blocks, in the reference's order per block, and shades them 32 at a time, one per
 * lane (resolve_item).
 */
#include "sftg_types.h"
#include "sftg_lane.cuh"
#include "sftg_kernels.h"

#define TILE_THREADS 256          /* resolve CTA */
#define RASTER_THREADS 512        /* raster CTA: 64 groups of 8 */
#define RASTER_BANDS 4            /* most row bands of a tile */
/* keys of one sample plane in shared memory: a whole tile, except at 4x, where every tile takes at
 * least 2 bands so that the keys (S x 32 KB per tile) leave room for 2 CTAs per SM */
template <int S> struct raster_plan {
    static constexpr int min_bands = S == 4 ? 2 : 1, plane = SFTG_TILE_PX / min_bands, rows = SFTG_TILE / min_bands;
};
#define SETUP_CAP RASTER_THREADS  /* triangle set-ups per round: one per thread */
#define MIN_SLAB_ROWS 4           /* smallest raster work item (rows); the slab height is a tuning knob */

struct tri_setup {
    float A[3], B[3], se[3];
    float sz, dzdx, dzdy;
    float pad[3];
    int ax0, ax1, miny, maxy;
    uint32_t order;
    int trivial;
};

/* tri_setup as kept in shared memory (56 B): the guard-band pads are recomputed from A and B,
 * the bounds are tile-local bytes (0..64) and the trivial-accept flag rides in order's top bit
 * (order = list position * 8 + lane stays below 2^31) */
struct tri_setup_packed {
    float A[3], B[3], se[3];
    float sz, dzdx, dzdy;
    uint32_t bounds;       /* ax0 | ax1 << 8 | miny << 16 | maxy << 24, tile-local */
    uint32_t order_triv;
};

SFTG_D tri_setup_packed pack_setup(const tri_setup& T, int tmx, int tmy) {
    tri_setup_packed P;
#pragma unroll
    for (int k = 0; k < 3; k++) { P.A[k] = T.A[k]; P.B[k] = T.B[k]; P.se[k] = T.se[k]; }
    P.sz = T.sz; P.dzdx = T.dzdx; P.dzdy = T.dzdy;
    P.bounds = (uint32_t)(T.ax0 - tmx) | ((uint32_t)(T.ax1 - tmx) << 8) | ((uint32_t)(T.miny - tmy) << 16) | ((uint32_t)(T.maxy - tmy) << 24);
    P.order_triv = T.order | (T.trivial ? 0x80000000u : 0u);
    return P;
}

template <int S>
SFTG_D tri_setup unpack_setup(const tri_setup_packed& P, int tmx, int tmy) {
    tri_setup T;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        T.A[k] = P.A[k]; T.B[k] = P.B[k]; T.se[k] = P.se[k];
        T.pad[k] = S > 1 ? 0.375f * (fabsf(P.A[k]) + fabsf(P.B[k])) : 0.f;   /* as in tri_setup_one */
    }
    T.sz = P.sz; T.dzdx = P.dzdx; T.dzdy = P.dzdy;
    T.ax0 = tmx + (int)(P.bounds & 0xFFu); T.ax1 = tmx + (int)((P.bounds >> 8) & 0xFFu);
    T.miny = tmy + (int)((P.bounds >> 16) & 0xFFu); T.maxy = tmy + (int)(P.bounds >> 24);
    T.order = P.order_triv & 0x7FFFFFFFu; T.trivial = (int)(P.order_triv >> 31);
    return T;
}

struct tri_verts {
    float sx[3], sy[3], iw[3], u[3], v[3], lu[3], lv[3], px[3], py[3], pz[3], nx[3], ny[3], nz[3];
    uint32_t inst, m;
};

__constant__ float c_ms_ox4[4] = { -0.125f, 0.375f, -0.375f, 0.125f };
__constant__ float c_ms_oy4[4] = { -0.375f, -0.125f, 0.125f, 0.375f };
__constant__ float c_ms_ox2[2] = { -0.25f, 0.25f };
__constant__ float c_ms_oy2[2] = { -0.25f, 0.25f };

template <int S> SFTG_D float ms_ox(int s) { return S == 4 ? c_ms_ox4[s] : (S == 2 ? c_ms_ox2[s] : 0.f); }
template <int S> SFTG_D float ms_oy(int s) { return S == 4 ? c_ms_oy4[s] : (S == 2 ? c_ms_oy2[s] : 0.f); }

/* a tile's depth range (1/w of its samples above 1e-4): the union of its raster bands' ranges */
SFTG_D float2 tile_zrange(const float2* zr, uint32_t gtile) {
    float2 r = zr[(size_t)gtile * RASTER_BANDS];
#pragma unroll
    for (int b = 1; b < RASTER_BANDS; b++) { const float2 q = zr[(size_t)gtile * RASTER_BANDS + b]; r.x = fminf(r.x, q.x); r.y = fmaxf(r.y, q.y); }
    return r;
}

SFTG_D uint64_t zkey(float z, uint32_t order) { return ((uint64_t)__float_as_uint(z) << 32) | (uint64_t)(0xFFFFFFFFu - order); }

/* vertices of one vis id (sofren2.c:5163-5209, 6199-6278) */
SFTG_D void fetch_tri(const sftg_tile_args& A, const sftg_inst* inst, const float* ss, const sftg_clip_tri* clips, uint32_t vid, tri_verts& t) {
    if (vid & 0x80000000u) {
        const sftg_clip_tri* c = &clips[vid & 0x7FFFFFFFu];
        const float* src = c->sx; float* dst = t.sx;
#pragma unroll
        for (int i = 0; i < 39; i++) dst[i] = src[i];
        t.inst = c->inst; t.m = c->m;
        return;
    }
    const uint32_t ii = (vid >> 25) & 63, m = (vid >> 7) & 0x3FFFF, tri = vid & 127;
    const sftg_inst* I = &inst[ii];
    const uint32_t g = I->meshlet_base + m;
    const uint8_t* ind = A.ml_inds + (size_t)g * 512;
    const float* Sc = ss + (size_t)(I->ss_offset + m) * SFTG_SS_FLOATS;
    const uint32_t b = tri >> 3, l = tri & 7;
    const uint32_t q[3] = { ind[b * 32 + l], ind[b * 32 + 8 + l], ind[b * 32 + 16 + l] };
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t v = q[k];
        const float4 a = ((const float4*)(Sc + SFTG_SS_A))[v], b4 = ((const float4*)(Sc + SFTG_SS_B))[v];
        const float4 c4 = ((const float4*)(Sc + SFTG_SS_C))[v];
        t.sx[k] = a.x; t.sy[k] = a.y; t.iw[k] = a.z;
        t.u[k] = c4.y; t.v[k] = c4.z; t.lu[k] = c4.w; t.lv[k] = Sc[SFTG_SS_D + v];
        t.px[k] = a.w; t.py[k] = b4.x; t.pz[k] = b4.y;
        t.nx[k] = b4.z; t.ny[k] = b4.w; t.nz[k] = c4.x;
    }
    t.inst = ii; t.m = m;
}

/* edge / depth setup of one triangle lane (5211-5311), false when culled or off-tile */
template <int S>
SFTG_D bool tri_setup_one(float sx0, float sy0, float iw0, float sx1, float sy1, float iw1, float sx2, float sy2, float iw2,
                          int tmx, int tmy, uint32_t order, tri_setup& T) {
    const float A0 = sy0 - sy1, B0 = sx1 - sx0, A1 = sy1 - sy2, B1 = sx2 - sx1, A2 = sy2 - sy0, B2 = sx0 - sx2;
    const float m01 = sx0 * sy1, m10 = sy0 * sx1, m12 = sx1 * sy2, m21 = sy1 * sx2, m20 = sx2 * sy0, m02 = sy2 * sx0;
    const float C0 = (fma_(sx0, sy1, -m10) - fma_(sy0, sx1, -m01)) * 0.5f;
    const float C1 = (fma_(sx1, sy2, -m21) - fma_(sy1, sx2, -m12)) * 0.5f;
    const float C2 = (fma_(sx2, sy0, -m02) - fma_(sy2, sx0, -m20)) * 0.5f;
    const float dx1 = sx1 - sx0, dx2 = sx2 - sx0, dy1 = sy1 - sy0, dy2 = sy2 - sy0;
    const float det = dx1 * dy2 - dx2 * dy1;
    if (!(det > 1e-6f)) return false;
    const float idet = rcpr(det);
    const float dzdx = ((iw1 - iw0) * dy2 - (iw2 - iw0) * dy1) * idet;
    const float dzdy = ((iw2 - iw0) * dx1 - (iw1 - iw0) * dx2) * idet;
    const float c0 = fma_(B0, 0.5f, fma_(A0, 0.5f, C0)), c1 = fma_(B1, 0.5f, fma_(A1, 0.5f, C1)), c2 = fma_(B2, 0.5f, fma_(A2, 0.5f, C2));
    const float zb = fma_(0.5f - sy0, dzdy, fma_(0.5f - sx0, dzdx, iw0));
    const int minx = cvtt(vmax(vmin(sx0, vmin(sx1, sx2)), (float)tmx));
    const int maxx = cvtt(vmin(vmax(sx0, vmax(sx1, sx2)), (float)(tmx + SFTG_TILE - 1)));
    const int miny = cvtt(vmax(vmin(sy0, vmin(sy1, sy2)), (float)tmy));
    const int maxy = cvtt(vmin(vmax(sy0, vmax(sy1, sy2)), (float)(tmy + SFTG_TILE - 1)));
    if (minx > maxx || miny > maxy) return false;
    const int ax0 = minx & ~7, ax1 = (maxx & ~7) + 8;
    T.A[0] = A0; T.A[1] = A1; T.A[2] = A2; T.B[0] = B0; T.B[1] = B1; T.B[2] = B2;
    T.se[0] = c0 + A0 * (float)ax0 + B0 * (float)miny;
    T.se[1] = c1 + A1 * (float)ax0 + B1 * (float)miny;
    T.se[2] = c2 + A2 * (float)ax0 + B2 * (float)miny;
    T.sz = zb + dzdx * (float)ax0 + dzdy * (float)miny;
    T.dzdx = dzdx; T.dzdy = dzdy;
    const float bw = (float)(ax1 - 1 - ax0), bh = (float)(maxy - miny);
    const float me0 = T.se[0] + (A0 < 0.f ? A0 * bw : 0.f) + (B0 < 0.f ? B0 * bh : 0.f);
    const float me1 = T.se[1] + (A1 < 0.f ? A1 * bw : 0.f) + (B1 < 0.f ? B1 * bh : 0.f);
    const float me2 = T.se[2] + (A2 < 0.f ? A2 * bw : 0.f) + (B2 < 0.f ? B2 * bh : 0.f);
    if (S > 1) {
        T.pad[0] = 0.375f * (fabsf(A0) + fabsf(B0));
        T.pad[1] = 0.375f * (fabsf(A1) + fabsf(B1));
        T.pad[2] = 0.375f * (fabsf(A2) + fabsf(B2));
        T.trivial = (me0 >= T.pad[0] && me1 >= T.pad[1] && me2 >= T.pad[2]);
    } else {
        T.pad[0] = T.pad[1] = T.pad[2] = 0.f;
        T.trivial = (me0 >= 0.f && me1 >= 0.f && me2 >= 0.f);
    }
    T.ax0 = ax0; T.ax1 = ax1; T.miny = miny; T.maxy = maxy; T.order = order;
    return true;
}

/* the least of three, NaN if one is: one instruction */
SFTG_D float min3(float a, float b, float c) { float r; asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
/* two floats in a register pair: one instruction adds both, each rounded as on its own */
typedef unsigned long long f32x2;
SFTG_D f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
SFTG_D float lo2(f32x2 v) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return a; }
SFTG_D float hi2(f32x2 v) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return b; }
SFTG_D f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

/* The incremental edge walk of one triangle's rows y0..y1 (5345-5497) by a group of 8 * S lanes: lane
 * (sample << 3 | l) owns one sample of pixel column l of every aligned 8-pixel chunk.  All lanes of a
 * column perform exactly the reference's adds of the pixel (row start + B per row, + 8A per chunk),
 * then each its own sample's offset.  Bound by issue: with 8 lanes per triangle and the samples in
 * turn, the four groups of a warp diverged over their triangles' sizes (17 of 32 threads) and the 4x
 * raster of the 1080p atrium took 0.287 ms; a warp per triangle 0.258, and 0.228 with slabs of 8 rows,
 * which now balance well enough (4 rows 0.251).  Of 50 instructions per step of a chunk: the trivial
 * triangles in a loop of their own, the least of the three edges instead of three comparisons, a vote
 * instead of a ballot and the step's adds in pairs took it to 0.197 (1279x719 1x 0.074 -> 0.062, skinned
 * 1080p 2x 0.090 -> 0.080, 48 views 3.41 -> 3.06); the row's adds in pairs too cost registers (2x 80
 * instead of 64, 48 views 3.9). */
template <int S>
SFTG_D void tri_raster(const tri_setup& T, int y0, int y1, int lane, uint32_t gmask, int tmx, int ky0, unsigned long long* keys) {
    const int l = lane & 7, smp = (lane >> 3) & (S - 1);
    const float ox = ms_ox<S>(smp), oy = ms_oy<S>(smp);
    const float de0 = T.A[0] * ox + T.B[0] * oy, de1 = T.A[1] * ox + T.B[1] * oy, de2 = T.A[2] * ox + T.B[2] * oy;
    const float dz = T.dzdx * ox + T.dzdy * oy;
    const float fl = (float)l;
    float e0r = T.se[0] + T.A[0] * fl, e1r = T.se[1] + T.A[1] * fl, e2r = T.se[2] + T.A[2] * fl;
    float zr = T.sz + T.dzdx * fl;
    /* a slab starting below miny replays the per-row adds it skips, so every row start is the
     * same float the reference's sequential walk reaches */
    for (int y = T.miny; y < y0; y++) { e0r = e0r + T.B[0]; e1r = e1r + T.B[1]; e2r = e2r + T.B[2]; zr = zr + T.dzdy; }
    const float a0c = T.A[0] * 8.f, a1c = T.A[1] * 8.f, a2c = T.A[2] * 8.f, zc = T.dzdx * 8.f;
    const float np0 = -T.pad[0], np1 = -T.pad[1], np2 = -T.pad[2];
    const uint32_t order = T.order;
    unsigned long long* const kp = keys + smp * raster_plan<S>::plane + (T.ax0 - tmx) + l;   /* keys hold the band's rows from ky0 */
    const int width = T.ax1 - T.ax0;
    if (T.trivial) {
        for (int y = y0; y <= y1; y++) {
            float z = zr;
            unsigned long long* k = kp + (y - ky0) * SFTG_TILE;
#pragma unroll 1
            for (int x = 0; x < width; x += 8, k += 8) {
                const float zs = (S > 1) ? z + dz : z;
                if (zs > 0.f) atomicMax(k, zkey(zs, order));
                z = z + zc;
            }
            zr = zr + T.dzdy;
        }
        return;
    }
    const f32x2 xA = pack2(a0c, a1c), xB = pack2(a2c, zc);
    unsigned long long* krow = kp + (y0 - ky0) * SFTG_TILE;
    for (int y = y0; y <= y1; y++, krow += SFTG_TILE) {
        f32x2 eA = pack2(e0r, e1r), eB = pack2(e2r, zr);
        unsigned long long* k = krow;
#pragma unroll 1
        for (int x = 0; x < width; x += 8, k += 8) {
            const float e0 = lo2(eA), e1 = hi2(eA), e2 = lo2(eB), z = hi2(eB);
            if (S == 1) {
                if (min3(e0, e1, e2) >= 0.f && z > 0.f) atomicMax(k, zkey(z, order));
            } else if (__any_sync(gmask, e0 >= np0 && e1 >= np1 && e2 >= np2)) {
                const float a = e0 + de0, b = e1 + de1, c = e2 + de2, zs = z + dz;
                if (min3(a, b, c) >= 0.f && zs > 0.f) atomicMax(k, zkey(zs, order));
            }
            eA = add2(eA, xA); eB = add2(eB, xB);
        }
        e0r = e0r + T.B[0]; e1r = e1r + T.B[1]; e2r = e2r + T.B[2]; zr = zr + T.dzdy;
    }
}

/* ---------------------------------------------------------------- texture sampling */
/* a texture's header and one level, a 16- and an 8-byte load */
struct tex_level { int w, h; bool pot; const uint32_t* base; uint32_t bw; };
SFTG_D tex_level tex_at(const sftg_tile_args& A, int4 head, int ti, int lod) {
    const uint2 lv = __ldg((const uint2*)&A.texs[ti].lev[lod]);
    tex_level t;
    t.w = max(head.x >> lod, 1); t.h = max(head.y >> lod, 1); t.pot = head.w != 0;
    t.base = A.texels + lv.x; t.bw = lv.y;
    return t;
}

SFTG_D uint32_t tex_addr(const tex_level& t, int u, int v) {
    const uint32_t uu = (uint32_t)u, vv = (uint32_t)v;
    return (((vv >> 2) * t.bw + (uu >> 2)) << 4) + ((vv & 3u) << 2) + (uu & 3u);
}

/* sft__sample_tex_bilinear (5543-5660), and sft__sample_tex_nearest (5662-5729) as the bilinear of one
 * texel: without the half-texel offset the corner is the nearest texel, and with zero fractions
 * f00 + (f10 - f00) * 0 is f00.  One code path, because a warp's lanes often need both. */
SFTG_D void sample_tex(const sftg_tile_args& A, int4 head, int ti, int lod, bool nearest, float cu, float cv, float& r, float& g, float& b) {
    if (ti < 0) { r = g = b = 1.f; return; }
    const tex_level t = tex_at(A, head, ti, lod);
    const int w = t.w, h = t.h;
    const float half = nearest ? 0.f : 0.5f;
    const float upx = cu * (float)w - half, vpx = cv * (float)h - half;
    const float uf0 = floorf(upx), vf0 = floorf(vpx);
    const float ufr = nearest ? 0.f : upx - uf0, vfr = nearest ? 0.f : vpx - vf0;
    const int u0 = cvtt(uf0), v0 = cvtt(vf0);
    const int wm = w - 1, hm = h - 1;
    int u0w, v0w, u1, v1;
    if (t.pot) { u1 = (u0 + 1) & wm; v1 = (v0 + 1) & hm; u0w = u0 & wm; v0w = v0 & hm; }
    else {   /* the reference's bilinear has no lower clamp here (it reads outside the texture); clamp at 0 */
        u1 = max(0, min(u0 + 1, wm)); v1 = max(0, min(v0 + 1, hm)); u0w = max(0, min(u0, wm)); v0w = max(0, min(v0, hm));
    }
    const uint32_t c00 = __ldg(&t.base[tex_addr(t, u0w, v0w)]);
    uint32_t c10 = c00, c01 = c00, c11 = c00;
    if (!nearest) { c10 = __ldg(&t.base[tex_addr(t, u1, v0w)]); c01 = __ldg(&t.base[tex_addr(t, u0w, v1)]); c11 = __ldg(&t.base[tex_addr(t, u1, v1)]); }
    const float i255 = 1.f / 255.f;
    float out[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int sh = 16 - 8 * k;
        const float f00 = (float)((c00 >> sh) & 255u) * i255, f10 = (float)((c10 >> sh) & 255u) * i255;
        const float f01 = (float)((c01 >> sh) & 255u) * i255, f11 = (float)((c11 >> sh) & 255u) * i255;
        const float top = f00 + (f10 - f00) * ufr, bot = f01 + (f11 - f01) * ufr;
        out[k] = top + (bot - top) * vfr;
    }
    r = out[0]; g = out[1]; b = out[2];
}

/* ---------------------------------------------------------------- raster */
/* One item, run by one CTA: its part of the tile's payload list into a shared-memory visibility buffer
 * (64-bit z/order words) for the band's rows, merged with the list's other parts where there are any,
 * then decoded into the global visibility buffer (float2: depth, vid bits) plus the band's depth
 * range over valid samples (sofren2.c:5820-5853), which the resolve needs for its light culling (a
 * tile's range is the union of its bands'). */
template <int S>
SFTG_D void raster_item(const sftg_tile_args& A, int slab_rows, const sftg_raster_item W)
{
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned long long* keys = (unsigned long long*)smem;                  /* S planes, a band uses the first band_px of each */
    tri_setup_packed* setups = (tri_setup_packed*)(smem + (size_t)S * raster_plan<S>::plane * 8);
    uint32_t* items = (uint32_t*)(setups + SETUP_CAP);                     /* set-up index << 8 | slab */
    __shared__ uint32_t s_nsetup, s_nbig, s_nsmall, s_next;
    /* work items of a round: long slabs from the front of the array, short ones from the back,
     * and the queue hands out the long ones first, so that a round does not end on one group
     * still walking a long slab (items touch keys only through atomicMax: order is free) */
    const uint32_t items_cap = (uint32_t)SETUP_CAP * (uint32_t)((raster_plan<S>::rows + slab_rows - 1) / slab_rows);
    __shared__ float s_red[2][RASTER_THREADS / 32];
    __shared__ uint32_t s_done;
    const uint32_t gtile = W.tile;   /* batch-wide tile index */
    const int band = W.band, bands = W.bands;
    const sftg_frame* F = A.frames + A.tile_view[gtile];
    const int tile = (int)(gtile - F->tile_base);
    const float* ss = A.ss + (size_t)F->ss_base * SFTG_SS_FLOATS;
    const sftg_clip_tri* clips = A.clips + (F->total_ss ? A.clip_base[F->ss_base] : 0u);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tmx = (tile % F->cols) * SFTG_TILE, tmy = (tile / F->cols) * SFTG_TILE;
    uint32_t count = A.tile_count[gtile];
    if ((uint64_t)A.tile_start[gtile] + count > F->tile_cap) count = 0;   /* overflowed frame, redone by the host */
    const int band_rows = SFTG_TILE / bands, band_px = band_rows * SFTG_TILE;
    const int by0 = tmy + band * band_rows, by1 = by0 + band_rows - 1;   /* this CTA's rows */
    const uint64_t* list = A.tile_pay + A.tile_start[gtile];
    float* vis_depth = A.vis_depth;
    uint32_t* vis_id = A.vis_id;

    for (int i = tid; i < S * band_px; i += RASTER_THREADS) keys[(i / band_px) * raster_plan<S>::plane + i % band_px] = 0ull;
    const int grp_lane = tid & 7;
    const uint32_t wmask = (0xFFFFFFFFu >> (32 - 8 * S)) << (lane & ~(8 * S - 1));   /* the walk's group */
    /* the payloads in equal rounds of at most SETUP_CAP / 8 (a short last round would leave most
     * groups idle at its barrier) */
    const uint32_t per_part = (count + W.parts - 1) / W.parts;
    const uint32_t part0 = min(count, W.part * per_part), part1 = min(count, part0 + per_part), mine = part1 - part0;
    const uint32_t rounds = (mine + SETUP_CAP / 8 - 1) / (SETUP_CAP / 8);
    const uint32_t per_round = rounds ? (mine + rounds - 1) / rounds : 1u;
    for (uint32_t pbase = part0; pbase < part1; pbase += per_round) {
        const uint32_t pend = min(part1, pbase + per_round);
        if (tid == 0) { s_nsetup = 0; s_nbig = 0; s_nsmall = 0; s_next = 0; }
        __syncthreads();
        {
            const uint32_t p = pbase + (tid >> 3);
            const int l = grp_lane;
            if (p < pend) {
                const uint64_t pay = list[p];
                const uint32_t raw = (uint32_t)(pay >> 56);
                float sx[3], sy[3], iw[3];
                bool active;
                if (!raw) {
                    active = (l == 0);
                    if (active) {
                        const sftg_clip_tri* c = &clips[(uint32_t)(pay & 0xFFFFFFFFu)];
#pragma unroll
                        for (int k = 0; k < 3; k++) { sx[k] = c->sx[k]; sy[k] = c->sy[k]; iw[k] = c->iw[k]; }
                    }
                } else {
                    active = (raw >> l) & 1u;
                    if (active) {
                        const uint32_t ii = (uint32_t)(pay & 0xFFFFFF), m = (uint32_t)((pay >> 24) & 0xFFFFFF), b = (uint32_t)((pay >> 48) & 0xFF);
                        const sftg_inst* I = &F->inst[ii];
                        const uint32_t g = I->meshlet_base + m;
                        const uint8_t* ind = A.ml_inds + (size_t)g * 512;
                        const float* Sc = ss + (size_t)(I->ss_offset + m) * SFTG_SS_FLOATS;
                        const uint32_t q[3] = { ind[b * 32 + l], ind[b * 32 + 8 + l], ind[b * 32 + 16 + l] };
#pragma unroll
                        for (int k = 0; k < 3; k++) { const float4 a = ((const float4*)(Sc + SFTG_SS_A))[q[k]]; sx[k] = a.x; sy[k] = a.y; iw[k] = a.z; }
                    }
                }
                if (active) {
                    tri_setup T;
                    /* the set-up is the whole tile's (bounds clamped to the 64x64 tile, edge values from
                     * its first row); the band keeps the triangles that reach its rows */
                    if (tri_setup_one<S>(sx[0], sy[0], iw[0], sx[1], sy[1], iw[1], sx[2], sy[2], iw[2], tmx, tmy, p * 8 + l, T) &&
                        T.maxy >= by0 && T.miny <= by1) {
                        const uint32_t slot = atomicAdd(&s_nsetup, 1u);
                        setups[slot] = pack_setup(T, tmx, tmy);
                        const int ys = max(T.miny, by0), ye = min(T.maxy, by1);
                        const uint32_t nslab = (uint32_t)(ye - ys) / (uint32_t)slab_rows + 1u;
                        const int rows = min(ye - ys + 1, slab_rows), chunks = (T.ax1 - T.ax0) >> 3;
                        if (S == 4 || rows * chunks >= 16) {   /* measured: the 4x raster keeps arrival order */
                            const uint32_t ib = atomicAdd(&s_nbig, nslab);
                            for (uint32_t k = 0; k < nslab; k++) items[ib + k] = (slot << 8) | k;
                        } else {
                            const uint32_t ib = atomicAdd(&s_nsmall, nslab);
                            for (uint32_t k = 0; k < nslab; k++) items[items_cap - 1u - (ib + k)] = (slot << 8) | k;
                        }
                    }
                }
            }
        }
        __syncthreads();
        const uint32_t nbig = s_nbig, nitem = nbig + s_nsmall;
        while (true) {
            uint32_t idx = 0;
            if ((lane & (8 * S - 1)) == 0) idx = atomicAdd(&s_next, 1u);
            idx = __shfl_sync(wmask, idx, lane & ~(8 * S - 1));
            if (idx >= nitem) break;
            const uint32_t it = idx < nbig ? items[idx] : items[items_cap - 1u - (idx - nbig)];
            const tri_setup T = unpack_setup<S>(setups[it >> 8], tmx, tmy);
            const int y0 = max(T.miny, by0) + (int)(it & 0xFFu) * slab_rows;   /* rows before y0 are replayed */
            const int y1 = min(y0 + slab_rows - 1, min(T.maxy, by1));
            tri_raster<S>(T, y0, y1, lane, wmask, tmx, by0, keys);
        }
        __syncthreads();
    }
    __syncthreads();
    float2* tv = A.vis + F->vis_base + (size_t)tile * S * SFTG_TILE_PX;
    unsigned long long* const merged = (unsigned long long*)tv;   /* of a list in parts: cleared by k_bin */
    if (W.parts > 1) {
        for (int i = tid; i < S * band_px; i += RASTER_THREADS) {
            const int sp = i / band_px, pp = i % band_px;
            const unsigned long long k = keys[sp * raster_plan<S>::plane + pp];
            if (k) atomicMax(&merged[sp * SFTG_TILE_PX + band * band_px + pp], k);
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) s_done = atomicAdd(&A.raster_done[gtile * RASTER_BANDS + band], 1u);
        __syncthreads();
        if (s_done + 1 != W.parts) return;   /* the last part decodes: nobody waits */
        __threadfence();
    }
    /* decode, store, depth range */
    float zmin = 1e9f, zmax = -1e9f;
    for (int i = tid; i < S * band_px; i += RASTER_THREADS) {
        const int sp = i / band_px, pp = i % band_px;
        const int ti = sp * SFTG_TILE_PX + band * band_px + pp;              /* the same sample in the tile */
        const unsigned long long k = W.parts > 1 ? __ldcg(&merged[ti]) : keys[sp * raster_plan<S>::plane + pp];
        float d = 0.f; uint32_t vid = SFTG_INVALID;
        if (k) {
            d = __uint_as_float((uint32_t)(k >> 32));
            const uint32_t order = 0xFFFFFFFFu - (uint32_t)k;
            const uint64_t pay = list[order >> 3];
            if ((pay >> 56) == 0) vid = (uint32_t)pay | 0x80000000u;
            else vid = ((uint32_t)(pay & 0xFFFFFF) << 25) | ((uint32_t)((pay >> 24) & 0xFFFFFF) << 7) | ((uint32_t)((pay >> 48) & 0xFF) * 8 + (order & 7));
        }
        tv[ti] = make_float2(d, __uint_as_float(vid));
        if (vis_id) {
            vis_depth[(size_t)tile * S * SFTG_TILE_PX + ti] = d;
            vis_id[(size_t)tile * S * SFTG_TILE_PX + ti] = vid;
        }
        if (d > 0.0001f) { zmin = fminf(zmin, d); zmax = fmaxf(zmax, d); }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) { zmin = fminf(zmin, __shfl_xor_sync(0xFFFFFFFFu, zmin, o)); zmax = fmaxf(zmax, __shfl_xor_sync(0xFFFFFFFFu, zmax, o)); }
    if (lane == 0) { s_red[0][warp] = zmin; s_red[1][warp] = zmax; }
    __syncthreads();
    if (tid == 0) {
        zmin = 1e9f; zmax = -1e9f;
        for (int w = 0; w < RASTER_THREADS / 32; w++) { zmin = fminf(zmin, s_red[0][w]); zmax = fmaxf(zmax, s_red[1][w]); }
        A.zrange[(size_t)gtile * RASTER_BANDS + band] = make_float2(zmin, zmax);   /* combined by the readers */
        if (band == 0) for (int b = bands; b < RASTER_BANDS; b++) A.zrange[(size_t)gtile * RASTER_BANDS + b] = make_float2(1e9f, -1e9f);
    }
}

/* one CTA per item; the grid is the bound on their number */
template <int S>
__global__ void __launch_bounds__(RASTER_THREADS)
k_raster(const sftg_tile_args A, int slab_rows)
{
    constexpr int si = S == 4 ? 2 : S - 1;
    if (blockIdx.x >= A.raster_range[3 + si]) return;
    raster_item<S>(A, slab_rows, A.raster_items[A.raster_range[si] + blockIdx.x]);
}

/* Persistent form: as many CTAs as fit on the GPU at once, each taking the next item in launch order
 * from a counter until all are taken.  The loop ends after at most items + grid counter reads:
 * nothing waits on another CTA. */
template <int S>
__global__ void __launch_bounds__(RASTER_THREADS, 2)   /* the 64 registers k_raster gets: 2 CTAs per SM */
k_raster_queue(const sftg_tile_args A, int slab_rows, uint32_t* next)
{
    constexpr int si = S == 4 ? 2 : S - 1;
    __shared__ uint32_t s_item;
    for (;;) {
        __syncthreads();   /* the previous item is done with shared memory, and s_item has been read */
        if (threadIdx.x == 0) s_item = atomicAdd(next, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= A.raster_range[3 + si]) break;
        raster_item<S>(A, slab_rows, A.raster_items[A.raster_range[si] + item]);
    }
}

/* ---------------------------------------------------------------- resolve */
/* D2 (5855-5934), one warp: the first SFTG_MAX_TILE_LIGHTS point lights in index order whose
 * depth range meets the tile's [zmin, zmax] and whose screen rectangle meets the tile.  Their
 * indices go to out[]; returns their count on every lane. */
SFTG_D int tile_light_list(const sftg_frame* F, float zmin, float zmax, int tmx, int tmy, int lane, uint16_t* out)
{
    int n = 0;
    if (zmin <= zmax && F->n_point > 0) {
        const float* vp = F->vp;
        for (uint32_t base = 0; base < F->n_point && n < SFTG_MAX_TILE_LIGHTS; base += 32) {
            const uint32_t l = base + lane;
            bool pass = false;
            if (l < F->n_point) {
                const sftg_point_light L = F->point[l];
                const float w = L.pos[0] * vp[3] + L.pos[1] * vp[7] + L.pos[2] * vp[11] + vp[15];
                const float lmin = w - L.radius, lmax = w + L.radius;
                pass = !(lmax <= 1e-6f);
                if (pass) {
                    const float smin = (lmin > 1e-6f) ? lmin : 1e-6f;
                    const float iwmin = fdiv(1.f, lmax), iwmax = fdiv(1.f, smin);
                    if (iwmax < zmin || iwmin > zmax) pass = false;
                }
                if (pass && w > L.radius) {
                    const float tx = L.pos[0] * vp[0] + L.pos[1] * vp[4] + L.pos[2] * vp[8] + vp[12];
                    const float ty = L.pos[0] * vp[1] + L.pos[1] * vp[5] + L.pos[2] * vp[9] + vp[13];
                    const float sx = (fdiv(tx, w) + 1.f) * F->hw + F->vpx;
                    const float sy = (fdiv(-ty, w) + 1.f) * F->hh + F->vpy;
                    const float psx = fsqrt(vp[0] * vp[0] + vp[4] * vp[4] + vp[8] * vp[8]);
                    const float psy = fsqrt(vp[1] * vp[1] + vp[5] * vp[5] + vp[9] * vp[9]);
                    const float safe_w = (w - L.radius) > 1e-6f ? (w - L.radius) : 1e-6f;
                    const float rx = fdiv((L.radius * psx) + fabsf(tx) * fdiv(L.radius, w), safe_w) * F->hw;
                    const float ry = fdiv((L.radius * psy) + fabsf(ty) * fdiv(L.radius, w), safe_w) * F->hh;
                    if (sx + rx < (float)tmx || sx - rx > (float)(tmx + SFTG_TILE) || sy + ry < (float)tmy || sy - ry > (float)(tmy + SFTG_TILE)) pass = false;
                }
            }
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, pass);
            const int rank = __popc(bal & ((1u << lane) - 1u));
            if (pass && n + rank < SFTG_MAX_TILE_LIGHTS) out[n + rank] = (uint16_t)l;
            n = min(SFTG_MAX_TILE_LIGHTS, n + __popc(bal));
        }
    }
    return n;
}

/* Per tile, once for all of its resolve CTAs: the light list (D2) and, per listed light, the
 * selected proxies (D3: in index order, those whose light_vis entry is set and whose bounding
 * sphere reaches the light's sphere, the first SFTG_MAX_LIGHT_PROXIES). */
__global__ void __launch_bounds__(TILE_THREADS)
k_tile_lights(const sftg_tile_args A, uint32_t tile0)
{
    __shared__ uint16_t s_lights[SFTG_MAX_TILE_LIGHTS];
    __shared__ int s_nlights;
    const uint32_t gtile = A.tile_order[tile0 + blockIdx.x];
    const sftg_frame* F = A.frames + A.tile_view[gtile];
    const int tile = (int)(gtile - F->tile_base);
    const uint8_t* light_vis = A.light_vis + (size_t)F->prox_base * 64;
    sftg_tile_lights* TL = A.tile_lights + gtile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tmx = (tile % F->cols) * SFTG_TILE, tmy = (tile / F->cols) * SFTG_TILE;
    const float2 zr = tile_zrange(A.zrange, gtile);
    const float zmin = zr.x, zmax = zr.y;

    if (warp == 0) {   /* D2 */
        const int n = tile_light_list(F, zmin, zmax, tmx, tmy, lane, s_lights);
        if (lane == 0) {
            s_nlights = n;
            A.tile_nlights[gtile] = (uint8_t)n;
            TL->nlights = (uint32_t)n;
        }
    }
    __syncthreads();
    const int ntl = s_nlights;
    if (tid < SFTG_MAX_TILE_LIGHTS) TL->light[tid] = tid < ntl ? s_lights[tid] : (uint16_t)0;
    for (int i = warp; i < SFTG_MAX_TILE_LIGHTS; i += TILE_THREADS / 32) {
        int n = 0;
        if (i < ntl && F->shadows && F->n_proxies > 0) {
            const sftg_point_light L = F->point[s_lights[i]];
            for (uint32_t base = 0; base < F->n_proxies && n < SFTG_MAX_LIGHT_PROXIES; base += 32) {
                const uint32_t p = base + lane;
                bool take = false;
                if (p < F->n_proxies && light_vis[(size_t)p * 64 + s_lights[i]]) {
                    const sftg_proxy px = F->proxies[p];
                    const v3 cc = mk3((px.posa[0] + px.posb[0]) * 0.5f, (px.posa[1] + px.posb[1]) * 0.5f, (px.posa[2] + px.posb[2]) * 0.5f);
                    const v3 ab = mk3(px.posb[0] - px.posa[0], px.posb[1] - px.posa[1], px.posb[2] - px.posa[2]);
                    const float cl = fsqrt(sdot(ab, ab));
                    const float br = px.radius + (cl * 0.5f);
                    const float cr = br + L.radius;
                    const v3 Wv = sub3(cc, mk3(L.pos[0], L.pos[1], L.pos[2]));
                    take = sdot(Wv, Wv) <= cr * cr;
                }
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, take);
                const int rank = __popc(bal & ((1u << lane) - 1u));
                if (take && n + rank < SFTG_MAX_LIGHT_PROXIES) TL->proxy[i][n + rank] = p;
                n = min(SFTG_MAX_LIGHT_PROXIES, n + __popc(bal));
            }
        }
        if (lane == 0) TL->npc[i] = (uint8_t)n;
    }
}

/* the batch exceeded a capacity: the host grows it and renders the batch again */
SFTG_D bool over_capacity(const sftg_tile_args& A, const sftg_frame* F) {
    return A.totals[0] > F->clip_cap || A.totals[1] > F->tile_cap || A.totals[2] > F->stile_cap;
}

#define TILE_BLOCKS (16 * 32)                 /* 4x2 blocks per 64x64 tile; a CTA resolves 1/split of them */
#define RESOLVE_WARPS (TILE_THREADS / 32)
#define LIGHT_SLOTS (SFTG_MAX_TILE_LIGHTS * SFTG_MAX_LIGHT_PROXIES)

/* A warp resolves `set` neighbouring 4x2 blocks at a time: up to max_set, fewer where a tile's
 * split leaves its 8 warps less (at 4x sets of 8 leave the L1 60 KB instead of 92: 0.336 ms against
 * 0.321 on the 1080p atrium, 0.161 against 0.136 at 155x106).  Its fragments (covered pixel, distinct
 * triangle) number at most max_set * 8 * S; a chunk of 32 is closed when the next (block, triangle)
 * pair does not fit, so it holds at least 25 of them, which bounds the chunks. */
template <int S> struct resolve_plan {
    static constexpr int max_set = S == 1 ? 16 : S == 2 ? 8 : 4;
    static constexpr int pixels = max_set * 8, chunks = pixels * S / 25 + 2, cap = chunks * 32;
};

/* A fragment: bits 0-2 pixel of its 4x2 block, 3-6 block of the set, 7-9 samples hit, 10-11 how
 * many triangles of the block covered this pixel before it, 12-16 lane where its (block, triangle)
 * pair starts, 17-24 the pair's covered pixels; FRAG_NONE pads a chunk. */
#define FRAG_NONE 0x80000000u

/* the OR of v over the lanes [start, end) of this lane's pair (at most 8 lanes, any offset) */
SFTG_D uint32_t pair_or(uint32_t v, int lane, int start, int end) {
    uint32_t t = __shfl_down_sync(0xFFFFFFFFu, v, 1); if (lane + 1 < end) v |= t;
    t = __shfl_down_sync(0xFFFFFFFFu, v, 2); if (lane + 2 < end) v |= t;
    t = __shfl_down_sync(0xFFFFFFFFu, v, 4); if (lane + 4 < end) v |= t;
    return __shfl_sync(0xFFFFFFFFu, v, start);
}

SFTG_D float warp_min(float v) { float r; asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v)); return r; }
SFTG_D float warp_max(float v) { float r; asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v)); return r; }

/* Bound by instruction issue.  With 8 lanes on each (block, triangle) pair, covered or not, 24 of 32
 * threads were active and a frame of few tiles waited for the block with the most triangles; a
 * lane per covered fragment and the proxies selected per 32 fragments instead of per CTA (which
 * also took a second interpolation of every pixel) measured: skinned characters 1080p 2x 0.252 ->
 * 0.172 ms, atrium 1080p 4x 0.541 -> 0.381, atrium 1279x719 1x 0.272 -> 0.103, mixed materials
 * 1333x717 2x 0.213 -> 0.143, skinned 320x180 2x 0.516 -> 0.074, a batch of 48 views 12.3 -> 8.0; with
 * the resident tables as kernel parameters, a texture's fields in two loads, a light's share of the
 * chunk's proxy filter computed once and no normals for lightmapped chunks 0.344 (4x) and 7.2.  Then
 * one issue slot in seven went to waits for instructions and one in three to loads that missed a small
 * L1: less code (three interpolations in one loop, one sampler, no branches in rcp and rsqrt), sets of 4
 * blocks at 4x (46 -> 33 KB of shared memory per CTA), sets handed out to the CTA's warps and a round's
 * places from one ballot gave 4x 0.303, 2x 0.172 -> 0.160 and 6.7 for the 48 views; a copy of the shading
 * of its own for `full` 2x 0.151, 6.5 and mixed materials 0.137 -> 0.131.
 * Sets of 16 blocks at 2x cost 3-15 %, contiguous sets per CTA at 4x 7 %.
 *
 * One (tile, part) item, run by one CTA.  The CTA makes the tile's light list and proxy cache
 * (5855-5990); then each warp resolves its sets of 4x2 blocks on its own (6029-6745):
 *   peel     one 8-thread group per block finds the block's distinct triangles in the reference's
 *            order and appends a fragment per covered pixel to the warp's list, four blocks at once
 *   shade    a lane per fragment, 32 at a time.  The reference shades the block's 8 pixels for
 *            every triangle; only covered pixels reach the image, and what the block shares is the
 *            LOD (the first covered pixel's derivatives: its neighbours' texture coordinates come
 *            from their lanes or are interpolated again) and the set of proxies that some covered
 *            pixel's segment to the light comes near (an OR over the pair's lanes)
 *   blend    a pixel's fragments follow one another in peel order, so the MSAA sum is accumulated
 *            in the reference's order
 * Uncovered pixels also keep a light from being skipped for their block.  That shows only where a
 * covered pixel's zero attenuation meets a value that is not finite (a light's colour, a proxy of
 * zero size, an interpolated position): such chunks are shaded again 8 lanes per pair, the
 * uncovered pixels among them, as the reference does (`full` below). */
template <bool B> struct flag_t { static constexpr bool value = B; };
template <int S>
SFTG_D void resolve_item(const sftg_tile_args& A, uint32_t tile0, int split, bool records, uint32_t item)
{
    using plan = resolve_plan<S>;
    /* proxy cache, entry light * 16 + slot: pa with |ab|^2, ab with radius^2, visibility factor; for
     * the per-lane "between" test W (proxy centre minus light) with |W|^2 and the squared bounding
     * radius; for the chunk filter the bounding radius grown by its share of the rounding margin */
    __shared__ float4 s_pa[LIGHT_SLOTS], s_ab[LIGHT_SLOTS], s_btw[LIGHT_SLOTS];
    __shared__ float s_vm[LIGHT_SLOTS], s_rb2[LIGHT_SLOTS], s_rbm[LIGHT_SLOTS];
    __shared__ uint16_t s_lights[SFTG_MAX_TILE_LIGHTS];
    __shared__ float4 s_lp[SFTG_MAX_TILE_LIGHTS], s_lc[SFTG_MAX_TILE_LIGHTS];   /* position with 1/r^2, colour */
    __shared__ int s_nlights, s_odd, s_set;
    __shared__ uint8_t s_npc[SFTG_MAX_TILE_LIGHTS];
    __shared__ uint32_t s_meta[RESOLVE_WARPS][plan::cap], s_vid[RESOLVE_WARPS][plan::cap];
    __shared__ float s_acc[RESOLVE_WARPS][S > 1 ? plan::pixels * 3 : 1];
    __shared__ uint32_t s_wm[RESOLVE_WARPS][SFTG_MAX_TILE_LIGHTS / 2];
    /* per warp and light, of the chunk in hand: its centre minus the light with 1 / |.|^2, the filter's radius */
    __shared__ float4 s_fd[RESOLVE_WARPS][SFTG_MAX_TILE_LIGHTS];
    __shared__ float s_fr[RESOLVE_WARPS][SFTG_MAX_TILE_LIGHTS];

    const uint32_t gtile = A.tile_order[tile0 + item / (uint32_t)split];   /* batch-wide tile index, heaviest first */
    const int part = (int)(item % (uint32_t)split);
    const sftg_frame* F = A.frames + A.tile_view[gtile];
    const int tile = (int)(gtile - F->tile_base);
    const float* ss = A.ss + (size_t)F->ss_base * SFTG_SS_FLOATS;
    const sftg_clip_tri* clips = A.clips + (F->total_ss ? A.clip_base[F->ss_base] : 0u);
    const uint8_t* light_vis = A.light_vis + (size_t)F->prox_base * 64;
    const sftg_inst* inst = F->inst;
    uint32_t* color = F->color_dev;
    const int CP = F->pitch;   /* colour row stride in pixels (the caller's buffer when written directly) */
    float* shadow_out = A.shadow_out;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tmx = (tile % F->cols) * SFTG_TILE, tmy = (tile / F->cols) * SFTG_TILE;
    const float2* vis = A.vis + F->vis_base + (size_t)tile * S * SFTG_TILE_PX;

    if (!F->clear && over_capacity(A, F)) return;   /* the whole CTA: the caller's pixels stay for the next attempt */
    const sftg_tile_lights* TL = A.tile_lights + gtile;
    if (tid == 0) { s_odd = shadow_out != nullptr; s_set = RESOLVE_WARPS; }
    if (records) {   /* D2 and D3's selection come from the tile's record (k_tile_lights) */
        if (tid < SFTG_MAX_TILE_LIGHTS) { s_lights[tid] = TL->light[tid]; s_npc[tid] = TL->npc[tid]; }
        if (tid == 0) s_nlights = (int)TL->nlights;
    } else if (warp == 0) {   /* D2 */
        const float2 zr = tile_zrange(A.zrange, gtile);
        const int n = tile_light_list(F, zr.x, zr.y, tmx, tmy, lane, s_lights);
        if (lane == 0) {
            s_nlights = n;
            if (part == 0) A.tile_nlights[gtile] = (uint8_t)n;
        }
    }
    __syncthreads();
    const int ntl = s_nlights;
    /* `odd`: a light or proxy with which a product with zero could be other than zero */
    if (tid < ntl) {
        const sftg_point_light L = F->point[s_lights[tid]];
        s_lp[tid] = make_float4(L.pos[0], L.pos[1], L.pos[2], L.inv_radius_sqr);
        s_lc[tid] = make_float4(L.color[0], L.color[1], L.color[2], 0.f);
        if (!(fabsf(L.pos[0]) + fabsf(L.pos[1]) + fabsf(L.pos[2]) <= 1e15f && fabsf(L.color[0]) + fabsf(L.color[1]) + fabsf(L.color[2]) <= 1e30f &&
              L.inv_radius_sqr >= 0.f && L.inv_radius_sqr <= 1e30f)) s_odd = 1;
    }
    /* D3's cache entry of proxy p in slot t (5936-5990) */
    auto cache = [&](int t, const sftg_proxy& px, uint8_t vs, const sftg_point_light& L, v3 ab, v3 Wv, float br, float d2) {
        s_pa[t] = make_float4(px.posa[0], px.posa[1], px.posa[2], sdot(ab, ab));
        s_ab[t] = make_float4(ab.x, ab.y, ab.z, px.radius * px.radius);
        s_vm[t] = (float)vs * 0.3333333f;
        s_btw[t] = make_float4(Wv.x, Wv.y, Wv.z, d2);
        s_rb2[t] = br * br;
        s_rbm[t] = sqrtf(br * br) + 2e-3f * sqrtf(d2) + 1e-3f + 1e-6f * (fabsf(L.pos[0]) + fabsf(L.pos[1]) + fabsf(L.pos[2]));
        if (!(fabsf(px.posa[0]) + fabsf(px.posa[1]) + fabsf(px.posa[2]) + fabsf(px.posb[0]) + fabsf(px.posb[1]) + fabsf(px.posb[2]) <= 1e15f &&
              px.radius >= 1e-15f && px.radius <= 1e15f)) s_odd = 1;
    };
    if (records) {   /* the tile's selected proxies, one thread per (light, slot) */
        for (int t = tid; t < LIGHT_SLOTS; t += TILE_THREADS) {
            const int i = t / SFTG_MAX_LIGHT_PROXIES, k = t % SFTG_MAX_LIGHT_PROXIES;
            if (i >= ntl || k >= s_npc[i]) continue;
            const uint32_t p = TL->proxy[i][k];
            const sftg_point_light L = F->point[s_lights[i]];   /* s_lp is read only after the next barrier */
            const sftg_proxy px = F->proxies[p];
            const uint8_t vs = light_vis[(size_t)p * 64 + s_lights[i]];
            const v3 cc = mk3((px.posa[0] + px.posb[0]) * 0.5f, (px.posa[1] + px.posb[1]) * 0.5f, (px.posa[2] + px.posb[2]) * 0.5f);
            const v3 ab = mk3(px.posb[0] - px.posa[0], px.posb[1] - px.posa[1], px.posb[2] - px.posa[2]);
            const float br = px.radius + (fsqrt(sdot(ab, ab)) * 0.5f);
            const v3 Wv = sub3(cc, mk3(L.pos[0], L.pos[1], L.pos[2]));
            cache(t, px, vs, L, ab, Wv, br, sdot(Wv, Wv));
        }
    } else {
        /* D3: per light, the first 16 proxies that see it and can reach it (5936-5990) */
        for (int i = warp; i < SFTG_MAX_TILE_LIGHTS; i += RESOLVE_WARPS) {
            int n = 0;
            if (i < ntl && F->shadows && F->n_proxies > 0) {
                const sftg_point_light L = F->point[s_lights[i]];
                for (uint32_t base = 0; base < F->n_proxies && n < SFTG_MAX_LIGHT_PROXIES; base += 32) {
                    const uint32_t p = base + lane;
                    bool take = false; uint8_t vs = 0;
                    v3 ab, Wv; float br = 0.f, d2 = 0.f;
                    sftg_proxy px;
                    if (p < F->n_proxies) {
                        px = F->proxies[p];
                        vs = light_vis[(size_t)p * 64 + s_lights[i]];
                        if (vs) {
                            const v3 cc = mk3((px.posa[0] + px.posb[0]) * 0.5f, (px.posa[1] + px.posb[1]) * 0.5f, (px.posa[2] + px.posb[2]) * 0.5f);
                            ab = mk3(px.posb[0] - px.posa[0], px.posb[1] - px.posa[1], px.posb[2] - px.posa[2]);
                            const float cl = fsqrt(sdot(ab, ab));
                            br = px.radius + (cl * 0.5f);
                            const float cr = br + L.radius;
                            Wv = sub3(cc, mk3(L.pos[0], L.pos[1], L.pos[2]));
                            d2 = sdot(Wv, Wv);
                            take = d2 <= cr * cr;
                        }
                    }
                    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, take);
                    const int rank = __popc(bal & ((1u << lane) - 1u));
                    if (take && n + rank < SFTG_MAX_LIGHT_PROXIES) cache(i * SFTG_MAX_LIGHT_PROXIES + n + rank, px, vs, L, ab, Wv, br, d2);
                    n = min(SFTG_MAX_LIGHT_PROXIES, n + __popc(bal));
                }
            }
            if (lane == 0) s_npc[i] = (uint8_t)n;
        }
    }
    __syncthreads();

    const int W = F->width;
    const int sw = (int)(F->hw * 2.f), sh = (int)(F->hh * 2.f);
    const int lim_x = min(tmx + SFTG_TILE, sw), lim_y = min(tmy + SFTG_TILE, sh);
    const bool proxies = F->shadows && F->n_proxies > 0 && ntl > 0;
    const bool clear = F->clear != 0;
    const int gl = lane & 7, gshift = lane & ~7;
    const float inv_s = 1.f / (float)S;
    const float i255 = 1.f / 255.f;
    const int ix = gl & 3, iy = gl >> 2;
    const uint32_t cc = F->clear_color;
    uint32_t* const metas = s_meta[warp];
    uint32_t* const vidl = s_vid[warp];
    float* const accs = s_acc[warp];
    uint32_t* const wm = s_wm[warp];

    /* the CTA's 512 / split blocks in sets of `set`: a set is 2 or 4 blocks wide */
    const int set = min(plan::max_set, TILE_BLOCKS / RESOLVE_WARPS / split);   /* 4, 8 or 16: split is at most 16 */
    const int bw = set >= 8 ? 4 : 2, across = 16 / bw, bh = set / bw;
    const int nsets = TILE_BLOCKS / set / split;
    /* sets beyond the first go to whichever warp is free (the 48 views 7.20 -> 7.07 ms) */
    auto next_set = [&]() { int q = 0; if (lane == 0) q = atomicAdd(&s_set, 1); return __shfl_sync(0xFFFFFFFFu, q, 0); };
    for (int q0 = warp; q0 < nsets; q0 = next_set()) {
        const int q = S == 4 ? q0 * split + part : part * nsets + q0;
        const int X0 = tmx + (q % across) * bw * 4, Y0 = tmy + (q / across) * bh * 2;
        if (X0 >= lim_x || Y0 >= lim_y) continue;   /* whole warp */

        /* ---------------- peel ---------------- */
        int cur = 0;             /* list position, uniform over the warp */
        uint32_t stores = 0;     /* bit k: this lane's pixel of its k-th block is written at the end */
        for (int k = 0; k < set / 4; k++) {
            const int bl = k * 4 + (lane >> 3);
            const int x = X0 + (bl % bw) * 4, y = Y0 + (bl / bw) * 2;
            const int gx = x + ix, gy = y + iy;
            const bool inb = sw > gx && sh > gy && x < lim_x && y < lim_y;
            const int pind = (gy - tmy) * SFTG_TILE + (gx - tmx);
            uint32_t vids[S], open[S];
            int ecount = 0;
            uint32_t act = 0;
#pragma unroll
            for (int s = 0; s < S; s++) {
                vids[s] = __float_as_uint(vis[s * SFTG_TILE_PX + pind].y);
                const bool empty = vids[s] == SFTG_INVALID;
                open[s] = (__ballot_sync(0xFFFFFFFFu, !empty && inb) >> gshift) & 0xFFu;
                ecount += (empty && inb);
                act |= open[s];
            }
            if (S == 1) {
                if (clear && inb && vids[0] == SFTG_INVALID) color[gy * CP + gx] = cc;
            } else if (!act) {
                if (clear && inb) color[gy * CP + gx] = cc;
            } else {   /* the empty samples' share of the background */
                const float ew = (float)ecount * inv_s;
                float bg[3] = { 0.f, 0.f, 0.f };
                if (clear || (ew > 0.f && inb)) {
                    const uint32_t c = clear ? cc : color[gy * CP + gx];
                    bg[0] = (float)((c >> 16) & 0xFF) * i255; bg[1] = (float)((c >> 8) & 0xFF) * i255; bg[2] = (float)(c & 0xFF) * i255;
                }
#pragma unroll
                for (int c = 0; c < 3; c++) accs[(bl * 8 + gl) * 3 + c] = bg[c] * ew;
                stores |= (uint32_t)(clear ? inb : ((act >> gl) & 1u)) << k;
            }
            uint32_t nj = 0;     /* triangles that covered this pixel so far */
            while (__any_sync(0xFFFFFFFFu, act != 0)) {
                /* the group's next triangle: the first covered pixel of its first sample plane with any left */
                const bool have = act != 0;
                uint32_t vsel = vids[0], osel = open[0];
#pragma unroll
                for (int s = 1; s < S; s++) if (!osel) { osel = open[s]; vsel = vids[s]; }
                const uint32_t target = __shfl_sync(0xFFFFFFFFu, vsel, gshift + (have ? __ffs(osel) - 1 : 0));
                uint32_t mask = 0, hits = 0;
                act = 0;
#pragma unroll
                for (int s = 0; s < S; s++) {
                    const bool match = have && inb && vids[s] == target;
                    const uint32_t mb = (__ballot_sync(0xFFFFFFFFu, match) >> gshift) & 0xFFu;
                    open[s] &= ~mb; mask |= mb; act |= open[s];
                    hits += match;
                }
                /* places for the four groups' pairs; a pair does not straddle two chunks */
                const uint32_t cov = __ballot_sync(0xFFFFFFFFu, (mask >> gl) & 1u);
                int at;
                if ((cur & 31) + __popc(cov) <= 32) {
                    at = cur + __popc(cov & ((1u << gshift) - 1u));
                    cur += __popc(cov);
                } else {
                    at = 0;
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        const int ng = __popc(cov & (0xFFu << (8 * g)));
                        if ((cur & 31) + ng > 32) {
                            const int nx = (cur + 31) & ~31;
                            if (cur + lane < nx) metas[cur + lane] = FRAG_NONE;
                            cur = nx;
                        }
                        if (g == (lane >> 3)) at = cur;
                        cur += ng;
                    }
                }
                if ((mask >> gl) & 1u) {
                    const int pos = at + __popc(mask & ((1u << gl) - 1u));
                    metas[pos] = (uint32_t)gl | (uint32_t)bl << 3 | hits << 7 | nj << 10 | (uint32_t)(at & 31) << 12 | mask << 17;
                    vidl[pos] = target;
                    nj++;
                }
            }
        }
        if (cur & 31) {
            const int nx = (cur + 31) & ~31;
            if (cur + lane < nx) metas[cur + lane] = FRAG_NONE;
            cur = nx;
        }
        __syncwarp();

        /* ---------------- shade ---------------- */
        /* One chunk; with `full` four of its pairs, 8 lanes each, uncovered pixels among them.  True where it has
         * to be called again: with `full`, or for the next four pairs.  Two copies of the code, one of which hardly
         * ever runs. */
        auto chunk = [&](auto FULL, int c0, int pass) -> bool {
            constexpr bool full = decltype(FULL)::value;
            uint32_t meta = metas[c0 + lane];
            uint32_t vid;
            int start, end, pl, npass = 1;
            bool in_tri;
            if (!full) {
                in_tri = !(meta & FRAG_NONE);
                if (!in_tri) meta = metas[c0];     /* a padding lane repeats the first fragment, without effect */
                vid = vidl[in_tri ? c0 + lane : c0];
                start = in_tri ? (int)((meta >> 12) & 31u) : lane;
                end = in_tri ? start + __popc((meta >> 17) & 0xFFu) : lane + 1;
                pl = (int)(meta & 7u);
            } else {
                uint32_t lead = __ballot_sync(0xFFFFFFFFu, !(meta & FRAG_NONE) && ((meta >> 12) & 31u) == (uint32_t)lane);
                npass = (__popc(lead) + 3) / 4;
                int src = 0;
                bool have = false;
                for (int k = 0; k <= pass * 4 + (lane >> 3); k++) { have = lead != 0; if (have) src = __ffs(lead) - 1; lead &= lead - 1; }
                const uint32_t mask = (metas[c0 + src] >> 17) & 0xFFu;
                in_tri = have && ((mask >> gl) & 1u);
                meta = metas[c0 + src + (in_tri ? __popc(mask & ((1u << gl) - 1u)) : 0)];
                vid = vidl[c0 + src];
                start = gshift; end = gshift + 8;
                pl = gl;
            }
            const int bl = (int)((meta >> 3) & 15u);
            const int x = X0 + (bl % bw) * 4, y = Y0 + (bl / bw) * 2;
            const int gx = x + (pl & 3), gy = y + (pl >> 2);
            tri_verts T;
            fetch_tri(A, inst, ss, clips, vid, T);
            const int4 info = __ldg((const int4*)&A.ml_info[inst[T.inst].meshlet_base + T.m]);   /* bone, skin slot, material, lightmap */
            /* D6 barycentrics and perspective-correct interpolation (6282-6347) */
            const float dx1 = T.sx[1] - T.sx[0], dx2 = T.sx[2] - T.sx[0], dy1 = T.sy[1] - T.sy[0], dy2 = T.sy[2] - T.sy[0];
            const float idet = rcpr(dx1 * dy2 - dx2 * dy1);
            float bu, bv, bw_, w0, w1, w2;
            auto weights = [&](float px, float py) {
                const float pxs = px - T.sx[0], pys = py - T.sy[0];
                const float rbu = (pxs * dy2 - pys * dx2) * idet;
                const float rbv = (pys * dx1 - pxs * dy1) * idet;
                const float rbw = (1.f - rbu) - rbv;
                bu = rbu; bv = rbv; bw_ = rbw;
                if (S > 1) {
                    bu = vmax(0.f, rbu); bv = vmax(0.f, rbv); bw_ = vmax(0.f, rbw);
                    const float bs = rcpr(bu + (bv + bw_));
                    bu = bu * bs; bv = bv * bs; bw_ = bw_ * bs;
                }
                const float iz = fma_(bw_, T.iw[0], fma_(bu, T.iw[1], bv * T.iw[2]));
                const float z = rcpr(iz);
                w0 = (bw_ * T.iw[0]) * z; w1 = (bu * T.iw[1]) * z; w2 = (bv * T.iw[2]) * z;
            };
            /* material (6350-6382) */
            uint32_t base = 0xFFFFFFFFu; int ti = -1; float shin = 4.f;
            if (info.z >= 0) {
                const int4 mt = __ldg((const int4*)&A.mats[info.z]);
                ti = mt.x; base = (uint32_t)mt.y; shin = __int_as_float(mt.z);
            }
            if (F->debug_mode == 5) { ti = F->debug_tex; base = 0xFFFFFFFFu; }   /* checkerboard view (6373-6376) */
            int4 head = make_int4(0, 0, 0, 0);   /* the texture's width, height, levels, pot */
            if (ti >= 0) head = __ldg((const int4*)&A.texs[ti]);
#define INTERP(a) fma_(w0, (a)[0], fma_(w1, (a)[1], w2 * (a)[2]))
            /* D7 LOD from the first covered lane's derivatives (5501-5541): its neighbours' coordinates from
             * their lanes where the triangle covers them, else interpolated here */
            const uint32_t mask = (meta >> 17) & 0xFFu;
            const int fl = __ffs(mask) - 1;
            const bool ok_x = full || ((mask >> (fl ^ 1)) & 1u), ok_y = full || ((mask >> (fl ^ 4)) & 1u);
            float cu_x = 0.f, cv_x = 0.f, cu_y = 0.f, cv_y = 0.f;
            float cu = 0.f, cv = 0.f;   /* the last turn leaves the fragment's own, and its weights */
#pragma unroll 1   /* one copy of the code: unrolled, the kernel's instruction fetches cost 4 % */
            for (int k = __any_sync(0xFFFFFFFFu, ti >= 0 && !(ok_x && ok_y)) ? 0 : 2; k < 3; k++) {
                const int at = k == 0 ? fl ^ 1 : k == 1 ? fl ^ 4 : pl;
                weights(((float)x + 0.5f) + (float)(at & 3), ((float)y + 0.5f) + (float)(at >> 2));
                cu_x = cu_y; cv_x = cv_y; cu_y = cu; cv_y = cv;
                cu = INTERP(T.u); cv = INTERP(T.v);
            }
            const float clu = INTERP(T.lu), clv = INTERP(T.lv);
            const v3 P = mk3(INTERP(T.px), INTERP(T.py), INTERP(T.pz));
            /* normal and view direction: a lightmapped surface uses neither */
            const bool lm = info.w >= 0;
            v3 N = mk3(0.f, 0.f, 0.f), V = N;
            if (__any_sync(0xFFFFFFFFu, !lm)) {
                N = vnorm_fast(mk3(INTERP(T.nx), INTERP(T.ny), INTERP(T.nz)));
                V = vnorm_fast(sub3(mk3(F->cam[0], F->cam[1], F->cam[2]), P));
            }
#undef INTERP
            if (!full && __any_sync(0xFFFFFFFFu, !(fabsf(P.x) + fabsf(P.y) + fabsf(P.z) <= 1e15f))) return true;
            bool wire = false;
            if (F->debug_mode == 1) {   /* wireframe view (6645-6671): edges where a barycentric is under its screen width */
                const float dbu_dx = (0.f - dy2) * idet, dbu_dy = dx2 * idet;
                const float dbv_dx = dy1 * idet, dbv_dy = (0.f - dx1) * idet;
                const float fw_u = fabsf(dbu_dx) + fabsf(dbu_dy), fw_v = fabsf(dbv_dx) + fabsf(dbv_dy);
                const float dbw_dx = 0.f - (dbu_dx + dbv_dx), dbw_dy = 0.f - (dbu_dy + dbv_dy);
                const float fw_w = fabsf(dbw_dx) + fabsf(dbw_dy);
                wire = bu < fw_u || bv < fw_v || bw_ < fw_w;
            }
            int lod = 0;
            {
                const int at_x = full ? gshift + (fl ^ 1) : start + __popc(mask & ((1u << (fl ^ 1)) - 1u));
                const int at_y = full ? gshift + (fl ^ 4) : start + __popc(mask & ((1u << (fl ^ 4)) - 1u));
                const int at_f = full ? gshift + fl : start;
                const float cu_f = __shfl_sync(0xFFFFFFFFu, cu, at_f), cv_f = __shfl_sync(0xFFFFFFFFu, cv, at_f);
                const float su_x = __shfl_sync(0xFFFFFFFFu, cu, at_x), sv_x = __shfl_sync(0xFFFFFFFFu, cv, at_x);
                const float su_y = __shfl_sync(0xFFFFFFFFu, cu, at_y), sv_y = __shfl_sync(0xFFFFFFFFu, cv, at_y);
                if (ok_x) { cu_x = su_x; cv_x = sv_x; }
                if (ok_y) { cu_y = su_y; cv_y = sv_y; }
                if (ti >= 0) {
                    const float ux = (cu_f - cu_x) * (float)head.x, vx = (cv_f - cv_x) * (float)head.y;
                    const float uy = (cu_f - cu_y) * (float)head.x, vy = (cv_f - cv_y) * (float)head.y;
                    const float a1 = fabsf(ux) > fabsf(vx) ? fabsf(ux) : fabsf(vx);
                    const float a2 = fabsf(uy) > fabsf(vy) ? fabsf(uy) : fabsf(vy);
                    const float rho = a1 > a2 ? a1 : a2;
                    if (rho > 1.f) {
                        const float lf = (float)(31 - __clz((uint32_t)cvtt(rho)));
                        lod = (int)((lf + 0.5f) + (-0.375f));
                    }
                    lod = lod < 0 ? 0 : (lod > head.z - 1 ? head.z - 1 : lod);
                }
            }
            float out[3];
            {
                float tr, tg, tb;
                sample_tex(A, head, ti, lod, lod > 1, cu, cv, tr, tg, tb);
                out[0] = tr * ((float)((base >> 16) & 0xFF) * i255); out[1] = tg * ((float)((base >> 8) & 0xFF) * i255);
                out[2] = tb * ((float)(base & 0xFF) * i255);
            }
            const bool lighted = !(shin < 0.f);
            if (!lighted) { out[0] = out[0] * (-shin); out[1] = out[1] * (-shin); out[2] = out[2] * (-shin); }
            if (__any_sync(0xFFFFFFFFu, lighted)) {
                const float sscale = ((shin + 8.f) / 8.f) * 0.04f;
                float dif[3], spc[3] = { 0.f, 0.f, 0.f }, lms = 1.f;
                if (lm) {
                    sample_tex(A, __ldg((const int4*)&A.texs[info.w]), info.w, 0, false, clu, clv, dif[0], dif[1], dif[2]);
                    dif[0] = dif[0] * F->lightmap_brightness; dif[1] = dif[1] * F->lightmap_brightness; dif[2] = dif[2] * F->lightmap_brightness;
                } else {
                    dif[0] = F->ambient[0]; dif[1] = F->ambient[1]; dif[2] = F->ambient[2];
                    for (uint32_t dl = 0; dl < F->n_dir; dl++) {
                        const sftg_dir_light D = F->dir[dl];
                        const v3 Ld = mk3(D.dir[0], D.dir[1], D.dir[2]);
                        const float ndl = vmax(vdot(N, Ld), 0.f);
                        dif[0] = fma_(ndl, D.color[0], dif[0]); dif[1] = fma_(ndl, D.color[1], dif[1]); dif[2] = fma_(ndl, D.color[2], dif[2]);
                        if (ndl > 0.f) {
                            const v3 Hh = vnorm_fast(add3(Ld, V));
                            const float ndh = vmax(vdot(N, Hh), 0.f);
                            const float den = (shin - shin * ndh) + ndh;
                            const float sp = ndh * rcpr(den);
                            const float term = (sp * sscale) * ndl;
                            spc[0] = fma_(term, D.color[0], spc[0]); spc[1] = fma_(term, D.color[1], spc[1]); spc[2] = fma_(term, D.color[2], spc[2]);
                        }
                    }
                }
                /* The chunk's own selection of the cached proxies, conservative: every shaded point lies in the
                 * ball (bc, br) around the chunk's bounds, so its segment to a light stays within br of the
                 * segment bc -> light, and a proxy farther than its bounding radius + br (+ a rounding margin)
                 * from that segment passes no pixel's "between" test (6520-6540).  Bit k of a light's 16: slot k. */
                uint32_t lb = ntl ? 0xFFFFFFFFu >> (32 - ntl) : 0u;   /* lights to visit */
                if (!full && ntl) {
                    uint32_t shadowing = 0;
                    if (proxies) {
                        const bool use = in_tri && lighted;
                        const float lx = warp_min(use ? P.x : 1e30f), ly = warp_min(use ? P.y : 1e30f), lz = warp_min(use ? P.z : 1e30f);
                        const float hx = warp_max(use ? P.x : -1e30f), hy = warp_max(use ? P.y : -1e30f), hz = warp_max(use ? P.z : -1e30f);
                        const v3 bc = mk3((lx + hx) * 0.5f, (ly + hy) * 0.5f, (lz + hz) * 0.5f);
                        const v3 he = mk3(hx - bc.x, hy - bc.y, hz - bc.z);
                        const float br = sqrtf(he.x * he.x + he.y * he.y + he.z * he.z) * 1.002f +
                                         1e-6f * (fabsf(bc.x) + fabsf(bc.y) + fabsf(bc.z));
                        if (lane < ntl) {
                            const float4 L = s_lp[lane];
                            const v3 D = mk3(bc.x - L.x, bc.y - L.y, bc.z - L.z);
                            const float dd = fma_(D.x, D.x, fma_(D.y, D.y, D.z * D.z));
                            s_fd[warp][lane] = make_float4(D.x, D.y, D.z, dd > 0.f ? __fdividef(1.f, dd) : 0.f);
                            s_fr[warp][lane] = br + (dd > 0.f ? 2e-3f * dd * rsqrtf(dd) : 0.f);
                        }
                        __syncwarp();
                        for (int i0 = 0; i0 < ntl; i0 += 2) {
                            const int i = i0 + (lane >> 4), k = lane & 15;
                            bool keep = false;
                            if (i < ntl && k < s_npc[i]) {
                                const float4 D = s_fd[warp][i], Wv = s_btw[i * SFTG_MAX_LIGHT_PROXIES + k];
                                const float t = __saturatef(fma_(Wv.x, D.x, fma_(Wv.y, D.y, Wv.z * D.z)) * D.w);
                                const v3 E = mk3(fma_(-t, D.x, Wv.x), fma_(-t, D.y, Wv.y), fma_(-t, D.z, Wv.z));
                                const float r = s_rbm[i * SFTG_MAX_LIGHT_PROXIES + k] + s_fr[warp][i];
                                keep = !(fma_(E.x, E.x, fma_(E.y, E.y, E.z * E.z)) > r * r);
                            }
                            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, keep);
                            if (lane == 0) wm[i0 >> 1] = bal;
                            shadowing |= ((bal & 0xFFFFu) ? 1u : 0u) << i0 | ((bal >> 16) ? 2u : 0u) << i0;
                        }
                        __syncwarp();
                    }
                    /* a light no proxy shadows leaves a lightmapped surface as it is */
                    if (__all_sync(0xFFFFFFFFu, lm || !in_tri || !lighted)) lb = shadowing;
                }
                /* D10 point lights and capsule shadows (6474-6607) */
                while (lb) {
                    const int i = __ffs(lb) - 1;
                    lb &= lb - 1;
                    const float4 L = s_lp[i];
                    const v3 Lr = sub3(mk3(L.x, L.y, L.z), P);
                    const float d2 = vdot(Lr, Lr);
                    float att = vmax(0.f, fma_(-d2, L.w, 1.f));
                    att = att * att;
                    const bool alive = att > 0.f;
                    /* a covered pixel out of the light's reach gets nothing from it; with `full`, not skipped
                     * while any pixel of the block is in reach */
                    bool go = alive;
                    if (full) go = pair_or(alive, lane, start, end) != 0;
                    go = go && lighted;
                    if (!__any_sync(0xFFFFFFFFu, go && in_tri)) continue;
                    v3 Ln = mk3(0.f, 0.f, 0.f);
                    float ndl = 0.f;
                    bool lit = false;
                    Ln = vnorm_fast(Lr);
                    if (!lm) {
                        ndl = vmax(vdot(N, Ln), 0.f);
                        lit = (ndl > 0.f) && alive && in_tri && lighted;
                    }
                    /* every selected proxy's "between" test first, then the block-level skip as the OR over
                     * the pair's lanes */
                    uint32_t pm = !proxies ? 0u : full ? (1u << s_npc[i]) - 1u : (wm[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu;
                    uint32_t rmask = 0, bmask = 0;
                    const bool want = lm ? in_tri && lighted : lit;
                    if (pm && __any_sync(0xFFFFFFFFu, want)) {
                        const float rd2 = rcpr(d2);   /* the reference recomputes the same value per proxy */
                        const float nd2 = -d2;
                        /* The reference's test with wdv = 0 - dot(W, Lr): wdv > 0 && wdv < d2, then
                         * cd2 = fma(-wdv, wdv * rd2, |W|^2) < rb2.  With v = dot(W, Lr): wdv > 0 is
                         * v < 0 (both false for a zero or NaN v), wdv < d2 is v > -d2, and for such
                         * v, wdv = -v exactly, wdv * rd2 = -(v * rd2) (round to nearest is
                         * symmetric) and cd2 = fma(-v, v * rd2, |W|^2): the same bits. */
                        while (pm) {
                            const int pi = __ffs(pm) - 1;
                            pm &= pm - 1;
                            const float4 bt = s_btw[i * SFTG_MAX_LIGHT_PROXIES + pi];
                            const float v = vdot(mk3(bt.x, bt.y, bt.z), Lr);
                            const bool btw = v < 0.f && v > nd2;
                            const float cd2 = fma_(-v, v * rd2, bt.w);
                            rmask |= (uint32_t)(btw && (cd2 < s_rb2[i * SFTG_MAX_LIGHT_PROXIES + pi]) && want) << pi;
                        }
                        if (__any_sync(0xFFFFFFFFu, rmask != 0)) bmask = pair_or(rmask, lane, start, end);
                    }
                    float msh = 0.f;
                    if (bmask) {
                        const float lrl = fsqrt(d2);
                        const float bk = 0.2f, b4 = 0.25f / 0.2f;
                        /* the smooth-max blend over the surviving proxies in index order */
                        while (bmask) {
                            const int pi = __ffs(bmask) - 1;
                            bmask &= bmask - 1;
                            const float4 qa = s_pa[i * SFTG_MAX_LIGHT_PROXIES + pi], qb = s_ab[i * SFTG_MAX_LIGHT_PROXIES + pi];
                            const bool ray = (rmask >> pi) & 1u;
                            const v3 pa = mk3(qa.x, qa.y, qa.z), ab = mk3(qb.x, qb.y, qb.z);
                            const v3 ao = sub3(P, pa);
                            const float abl = vdot(ab, Ln), abao = vdot(ab, ao), lao = vdot(Ln, ao);
                            const float den = fma_(-abl, abl, qa.w);
                            const float sden = vmax(den, 1e-6f);
                            float t2 = fma_(-abl, lao, abao) * rcpr(sden);
                            t2 = vmax(0.f, vmin(t2, 1.f));
                            const float t1 = fma_(t2, abl, -lao);
                            const bool vc = t1 > 1e-6f && t1 < lrl;
                            const v3 pr = add3(P, scl3(Ln, t1));
                            const v3 pc = add3(pa, scl3(ab, t2));
                            const v3 dd = sub3(pr, pc);
                            const float dist2 = vdot(dd, dd);
                            float sv = vmax(0.f, 1.f - fdiv(dist2, qb.w));
                            if (!ray || !vc) sv = 0.f;
                            sv = sv * s_vm[i * SFTG_MAX_LIGHT_PROXIES + pi];
                            const float h = vmax(0.f, bk - fabsf(msh - sv));
                            const float badd = (h * h) * b4;
                            msh = vmax(msh, sv) + badd;
                        }
                    }
                    const float si = vmax(0.f, 1.f - msh);
                    if (S == 1 && shadow_out && go && in_tri && i < 16) shadow_out[((size_t)gy * W + gx) * 16 + i] = si;
                    if (lm) {
                        const float drop = (1.f - si) * att;
                        if (go) lms = lms * (1.f - drop);
                    } else if (lit || (full && go)) {
                        const float4 C = s_lc[i];
                        const float di = ndl * att;
                        const float md = lit ? (di * si) : 0.f;
                        dif[0] = fma_(md, C.x, dif[0]); dif[1] = fma_(md, C.y, dif[1]); dif[2] = fma_(md, C.z, dif[2]);
                        if (lit) {
                            const v3 Hh = vnorm_fast(add3(Ln, V));
                            const float ndh = vmax(vdot(N, Hh), 0.f);
                            const float den = (shin - shin * ndh) + ndh;
                            const float sp = ndh * rcpr(den);
                            const float term = ((sp * sscale) * di) * si;
                            spc[0] = fma_(term, C.x, spc[0]); spc[1] = fma_(term, C.y, spc[1]); spc[2] = fma_(term, C.z, spc[2]);
                        }
                    }
                }
                if (lighted) {
                    if (lm) {
                        const float mod = fma_(lms, 1.f - 0.4f, 0.4f);
                        out[0] = out[0] * (dif[0] * mod); out[1] = out[1] * (dif[1] * mod); out[2] = out[2] * (dif[2] * mod);
                    } else {
                        out[0] = fma_(out[0], dif[0], spc[0]); out[1] = fma_(out[1], dif[1], spc[1]); out[2] = fma_(out[2], dif[2], spc[2]);
                    }
                }
            }
            if (wire) { out[0] = 0.f; out[1] = 1.f; out[2] = 0.f; }
            if (S == 1) {
                if (in_tri) {
                    uint32_t px = 0xFF000000u;
#pragma unroll
                    for (int k = 0; k < 3; k++) px |= ((uint32_t)cvtt(vmax(0.f, vmin(out[k], 1.f)) * 255.f)) << (16 - 8 * k);
                    color[gy * CP + gx] = px;
                }
            } else {
                /* a pixel's fragments of one chunk are added in turn */
                const float wgt = (float)((meta >> 7) & 7u) * inv_s;
                const uint32_t j = (meta >> 10) & 3u;
                float* const a = accs + (bl * 8 + pl) * 3;
#pragma unroll
                for (uint32_t jj = 0; jj < (uint32_t)S; jj++) {
                    if (in_tri && j == jj)
#pragma unroll
                        for (int k = 0; k < 3; k++) a[k] = fma_(vmax(0.f, vmin(out[k], 1.f)), wgt, a[k]);
                    __syncwarp();
                }
            }
            return full && pass + 1 < npass;
        };
        const bool odd = s_odd != 0;
        for (int c0 = 0; c0 < cur; c0 += 32)
            if (odd || chunk(flag_t<false>(), c0, 0))
                for (int pass = 0; chunk(flag_t<true>(), c0, pass); pass++) { }

        /* ---------------- store ---------------- */
        if (S > 1) {
            for (int k = 0; k < set / 4; k++) {
                if (!((stores >> k) & 1u)) continue;
                const int bl = k * 4 + (lane >> 3);
                const int gx = X0 + (bl % bw) * 4 + ix, gy = Y0 + (bl / bw) * 2 + iy;
                const float* a = accs + (bl * 8 + gl) * 3;
                uint32_t px = 0xFF000000u;
#pragma unroll
                for (int c = 0; c < 3; c++) px |= ((uint32_t)cvtt(vmin(a[c], 1.f) * 255.f)) << (16 - 8 * c);
                color[gy * CP + gx] = px;
            }
        }
        __syncwarp();   /* the next set reuses the warp's list and sums */
    }
}

/* one CTA per (tile, part) item */
template <int S>
__global__ void __launch_bounds__(TILE_THREADS, 4)   /* 64 registers; 80 (3 CTAs) cost 2-7 %, 48 (5 CTAs) 5-11 % */
k_resolve(const sftg_tile_args A, uint32_t tile0, int split, bool records)
{
    resolve_item<S>(A, tile0, split, records, blockIdx.x);
}

/* Persistent form, as k_raster_queue: CTAs take (tile, part) items in launch order from a counter. */
template <int S>
__global__ void __launch_bounds__(TILE_THREADS, 4)
k_resolve_queue(const sftg_tile_args A, uint32_t tile0, int split, bool records, uint32_t n_items, uint32_t* next)
{
    __shared__ uint32_t s_item;
    for (;;) {
        __syncthreads();   /* the previous item is done with shared memory, and s_item has been read */
        if (threadIdx.x == 0) s_item = atomicAdd(next, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= n_items) break;
        resolve_item<S>(A, tile0, split, records, item);
    }
}

/* ---------------------------------------------------------------- tile order
 * The reference's workers take tiles in descending payload count (sofren2.c:6815-6857) so the
 * heaviest start first.  Here the same idea keeps the tail of the raster and resolve grids
 * short: tiles are bucketed by floor(log2(count + 1)) inside their sample-count range and the
 * launches walk the buckets heaviest first.  Order affects scheduling only, never results. */
#define ORDER_BUCKETS 32
#define ORDER_ALL (3 * ORDER_BUCKETS)

__device__ __forceinline__ uint32_t order_bucket(const sftg_frame* frames, const uint16_t* tile_view, const uint32_t* tile_count, uint32_t t) {
    const int S = frames[tile_view[t]].samples;
    const uint32_t si = S == 1 ? 0u : (S == 2 ? 1u : 2u);
    const uint32_t key = 31u - (uint32_t)__clz(tile_count[t] + 1u);          /* 0..31, heavier = larger */
    return si * ORDER_BUCKETS + (ORDER_BUCKETS - 1u - key);
}

struct band_knobs { int b[3], whole; };   /* tuning.raster_bands; least bands of a list in one part */

/* row bands of a tile at 1x, 2x, 4x (slot si): the knob's, at 4x at least 2 (shared memory) */
__device__ __forceinline__ uint32_t order_bands(const band_knobs& K, uint32_t si, uint32_t parts) {
    const uint32_t b = (uint32_t)K.b[si], l = si == 2u ? 2u : 1u, w = parts == 1u ? (uint32_t)K.whole : 1u, least = l > w ? l : w;
    return b > least ? b : least;
}

/* Least bands of the tiles whose list is not cut, for a batch of few tiles: doubled while the tiles'
 * bands number fewer than the resident CTAs.  A short list can hold triangles that fill the tile, which
 * rows divide without the merge that parts need: mixed materials 1333x717 2x (252 tiles, 2 bands) 0.092
 * -> 0.070 ms, 4 bands 0.097; atrium 1280x720 2x (240 tiles) 0.162 -> 0.148; parts of 4 payloads instead
 * 0.082, and they cost a 640x360 frame of 60 tiles 0.010 where bands cost nothing. */
static int whole_bands(uint32_t tiles) {
    int b = 1;
    while (b < RASTER_BANDS && tiles * (uint32_t)b < SFTG_RASTER_CTAS) b *= 2;
    return b;
}

/* the exclusive starts of both histograms, and the item range of every sample count */
__device__ __forceinline__ void order_starts(const uint32_t* h, uint32_t* base, uint32_t* range) {
    uint32_t run = 0, items = 0;
    for (uint32_t i = 0; i < ORDER_ALL; i++) {
        if (range && i % ORDER_BUCKETS == 0) range[i / ORDER_BUCKETS] = items;
        base[i] = run; base[ORDER_ALL + i] = items;
        run += h[i]; items += h[ORDER_ALL + i];
        if (range && i % ORDER_BUCKETS == ORDER_BUCKETS - 1) range[3 + i / ORDER_BUCKETS] = items - range[i / ORDER_BUCKETS];
    }
}

/* tile t's place in the order and its raster items, from counters that start at its bucket's */
__device__ __forceinline__ void order_place(uint32_t t, uint32_t b, uint32_t count, uint32_t total, const band_knobs& K, uint32_t* cursor,
                                            uint32_t* order, sftg_raster_item* items) {
    order[atomicAdd(&cursor[b], 1u)] = t;
    const uint32_t parts = sftg_raster_parts(count, total, 1 << (b / ORDER_BUCKETS)), bands = order_bands(K, b / ORDER_BUCKETS, parts);
    uint32_t at = atomicAdd(&cursor[ORDER_ALL + b], bands * parts);
    for (uint32_t p = 0; p < parts; p++)
        for (uint32_t k = 0; k < bands; k++) {
            sftg_raster_item w;
            w.tile = t; w.band = (uint8_t)k; w.bands = (uint8_t)bands; w.part = (uint16_t)p; w.parts = parts; w.pad = 0;
            items[at++] = w;
        }
}

__global__ void k_order_count(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ tile_view,
                              const uint32_t* __restrict__ tile_count, uint32_t n_tiles, const uint32_t* __restrict__ total,
                              const band_knobs K, uint32_t* __restrict__ hist)
{
    __shared__ uint32_t h[2 * ORDER_ALL];
    for (int i = threadIdx.x; i < 2 * ORDER_ALL; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_tiles) {
        const uint32_t b = order_bucket(frames, tile_view, tile_count, t);
        atomicAdd(&h[b], 1u);
        const uint32_t parts = sftg_raster_parts(tile_count[t], *total, 1 << (b / ORDER_BUCKETS));
        atomicAdd(&h[ORDER_ALL + b], order_bands(K, b / ORDER_BUCKETS, parts) * parts);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * ORDER_ALL; i += blockDim.x) if (h[i]) atomicAdd(&hist[i], h[i]);
}

/* one CTA: the starts, into the histogram's place */
__global__ void k_order_starts(uint32_t* __restrict__ hist, uint32_t* __restrict__ range)
{
    __shared__ uint32_t h[2 * ORDER_ALL], base[2 * ORDER_ALL];
    for (int i = threadIdx.x; i < 2 * ORDER_ALL; i += blockDim.x) h[i] = hist[i];
    __syncthreads();
    if (threadIdx.x == 0) order_starts(h, base, range);
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * ORDER_ALL; i += blockDim.x) hist[i] = base[i];
}

__global__ void k_order_scatter(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ tile_view,
                                const uint32_t* __restrict__ tile_count, uint32_t n_tiles, const uint32_t* __restrict__ total,
                                const band_knobs K, uint32_t* __restrict__ cursor, uint32_t* __restrict__ order,
                                sftg_raster_item* __restrict__ items)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_tiles) order_place(t, order_bucket(frames, tile_view, tile_count, t), tile_count[t], *total, K, cursor, order, items);
}

/* The whole of it in one CTA for small tile counts: the scan of the segments' counts (each thread a
 * run of them), every tile's count and start, then histogram, bucket starts and scatter.  One launch
 * between the binning's passes instead of a scan before and an order after the second. */
__global__ void __launch_bounds__(1024)
k_tile_starts(const sftg_frame* __restrict__ frames, const uint16_t* __restrict__ tile_view, const uint32_t* seg_count, uint32_t nseg,
              uint32_t n_tiles, uint32_t* seg_start, uint32_t* tile_count, uint32_t* tile_start, uint32_t* __restrict__ total,
              const band_knobs K, uint32_t* __restrict__ order, sftg_raster_item* __restrict__ items, uint32_t* __restrict__ range)
{
    __shared__ uint32_t h[2 * ORDER_ALL], base[2 * ORDER_ALL], s_w[32], s_all;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < 2 * ORDER_ALL; i += 1024) h[i] = 0;
    const uint32_t n = n_tiles * nseg, per = (n + 1023u) / 1024u, i0 = (uint32_t)tid * per;
    uint32_t sum = 0;
    for (uint32_t k = 0; k < per; k++) if (i0 + k < n) sum += seg_count[i0 + k];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o); if (lane >= o) incl += t; }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = s_w[lane];
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, wi, o); if (lane >= o) wi += t; }
        s_w[lane] = wi - w;
        if (lane == 31) { s_all = wi; *total = wi; }
    }
    __syncthreads();
    uint32_t at = s_w[warp] + incl - sum;
    for (uint32_t k = 0; k < per; k++) if (i0 + k < n) { seg_start[i0 + k] = at; at += seg_count[i0 + k]; }
    __syncthreads();
    const uint32_t all = s_all;
    for (uint32_t t = tid; t < n_tiles; t += 1024) {
        if (nseg > 1) {
            const uint32_t a = seg_start[t * nseg], e = t + 1 < n_tiles ? seg_start[(t + 1) * nseg] : all;
            tile_start[t] = a; tile_count[t] = e - a;
        }
        const uint32_t b = order_bucket(frames, tile_view, tile_count, t);
        atomicAdd(&h[b], 1u);
        const uint32_t parts = sftg_raster_parts(tile_count[t], all, 1 << (b / ORDER_BUCKETS));
        atomicAdd(&h[ORDER_ALL + b], order_bands(K, b / ORDER_BUCKETS, parts) * parts);
    }
    __syncthreads();
    if (tid == 0) order_starts(h, base, range);
    __syncthreads();
    for (uint32_t t = tid; t < n_tiles; t += 1024)
        order_place(t, order_bucket(frames, tile_view, tile_count, t), tile_count[t], all, K, base, order, items);
}

#define ORDER_SMALL 8192u   /* tile counts up to this are handled by one CTA */

bool sftg_launch_tile_starts(const sftg_frame* frames, const uint16_t* tile_view, const uint32_t* seg_count, uint32_t nseg, uint32_t n_tiles,
                             uint32_t* seg_start, uint32_t* tile_count, uint32_t* tile_start, uint32_t* total, const int* bands,
                             uint32_t* order, sftg_raster_item* items, uint32_t* range, cudaStream_t st, int* launches) {
    if (n_tiles > ORDER_SMALL) return false;
    const band_knobs K = { { bands[0], bands[1], bands[2] }, whole_bands(n_tiles) };
    k_tile_starts<<<1, 1024, 0, st>>>(frames, tile_view, seg_count, nseg, n_tiles, seg_start, tile_count, tile_start, total, K, order, items, range);
    *launches += 1;
    return true;
}

void sftg_launch_tile_order(const sftg_frame* frames, const uint16_t* tile_view, const uint32_t* tile_count, uint32_t n_tiles,
                            const uint32_t* total, const int* bands, uint32_t* scratch, uint32_t* order, sftg_raster_item* items,
                            uint32_t* range, cudaStream_t st, int* launches) {
    const band_knobs K = { { bands[0], bands[1], bands[2] }, whole_bands(n_tiles) };
    cudaMemsetAsync(scratch, 0, 2 * ORDER_ALL * sizeof(uint32_t), st);
    const uint32_t g = (n_tiles + 255) / 256;
    k_order_count<<<g, 256, 0, st>>>(frames, tile_view, tile_count, n_tiles, total, K, scratch);
    k_order_starts<<<1, 256, 0, st>>>(scratch, range);
    k_order_scatter<<<g, 256, 0, st>>>(frames, tile_view, tile_count, n_tiles, total, K, scratch, order, items);
    *launches += 3;
}

uint32_t sftg_raster_items_max(int S, uint32_t tiles, int bands) {
    const uint32_t least = S == 4 ? 2u : 1u, b = (uint32_t)bands > least ? (uint32_t)bands : least;
    const uint32_t w = (uint32_t)whole_bands(tiles), bw = b > w ? b : w;   /* of all the batch's tiles it is no larger */
    return bw * tiles + b * (tiles + 2u * SFTG_RASTER_CTAS);   /* uncut tiles; parts: one per tile, and one per share of the payloads */
}

/* ---------------------------------------------------------------- debug overlays
 * sft__debug_draw_tile_overlay (5731-5807): tile borders and a 16-pixel grid (view 2), sample-0
 * linear depth with a border coloured by the tile's depth span (view 3), a heat tint from the
 * tile's light count (view 4).  One CTA per tile, after every tile has been resolved; each
 * overlay touches only its own tile, as in the reference where it follows that tile's resolve. */
__device__ __forceinline__ uint32_t half_blend(uint32_t bg, uint32_t ov) { return ((bg & 0xFEFEFEFEu) >> 1) + ((ov & 0xFEFEFEFEu) >> 1); }

__global__ void __launch_bounds__(256) k_debug_overlay(const sftg_tile_args A)
{
    const uint32_t gtile = blockIdx.x;
    const sftg_frame* F = A.frames + A.tile_view[gtile];
    const int mode = F->debug_mode;
    if (mode < 2 || mode > 4) return;
    if (!F->clear && over_capacity(A, F)) return;
    const int tile = (int)(gtile - F->tile_base);
    const int tmx = (tile % F->cols) * SFTG_TILE, tmy = (tile / F->cols) * SFTG_TILE;
    const int sw = (int)(F->hw * 2.f), sh = (int)(F->hh * 2.f);
    const int lim_x = min(tmx + SFTG_TILE, sw), lim_y = min(tmy + SFTG_TILE, sh);
    uint32_t* color = F->color_dev;
    const float2* depth = A.vis + F->vis_base + (size_t)tile * F->samples * SFTG_TILE_PX;   /* sample 0 plane first */
    const float2 zr = tile_zrange(A.zrange, gtile);
    const int ntl = A.tile_nlights[gtile];
    uint32_t border = 0xFF00FF00u, heat = 0;
    if (mode == 3) {
        float dd = 0.f;
        if (zr.x <= zr.y && zr.x > 1e-6f) { const float near_w = fdiv(1.f, zr.y), far_w = fdiv(1.f, zr.x); dd = far_w - near_w; }
        border = dd > 16.f ? 0xFFFF0000u : 0xFF00FF00u;
    }
    if (mode == 4) heat = ntl == 0 ? 0xFF222288u : (ntl < 4 ? 0xFF00FF00u : 0xFFFF0000u);
    for (int i = threadIdx.x; i < SFTG_TILE_PX; i += blockDim.x) {
        const int x = tmx + (i & (SFTG_TILE - 1)), y = tmy + (i >> 6);
        if (x >= lim_x || y >= lim_y) continue;
        uint32_t* p = &color[(size_t)y * F->pitch + x];
        const bool edge = x == tmx || x == lim_x - 1 || y == tmy || y == lim_y - 1;
        if (mode == 2) {
            if (edge) *p = 0xFF00FF00u;
            else if ((x % 16 == 0) || (y % 16 == 0)) *p = half_blend(*p, 0xFF004400u);
        } else if (mode == 3) {
            if (edge) { *p = border; continue; }
            const float iw = depth[i].x;
            if (iw <= 1e-6f) continue;
            const float lz = fdiv(1.f, iw);
            const float q = fdiv(lz, 100.f);
            const float nz = q < 0.f ? 0.f : (q > 1.f ? 1.f : q);
            const uint32_t it = (uint32_t)(nz * 255.f);
            *p = 0xFF000000u | (it << 16) | (it << 8) | it;
        } else {
            *p = half_blend(*p, heat);
        }
    }
}

void sftg_launch_debug_overlay(uint32_t tiles, cudaStream_t st, const sftg_tile_args& A) {
    if (tiles) k_debug_overlay<<<tiles, 256, 0, st>>>(A);
}

/* ---------------------------------------------------------------- host-side launch helpers */
/* keys, packed set-ups, then the work items of one round: up to SETUP_CAP * (64 / slab_rows) */
static size_t raster_smem(int S, int slab_rows) {
    const size_t plane = S == 4 ? raster_plan<4>::plane : SFTG_TILE_PX, rows = S == 4 ? raster_plan<4>::rows : SFTG_TILE;
    return (size_t)S * plane * 8 + (size_t)SETUP_CAP * sizeof(tri_setup_packed) +
           (size_t)SETUP_CAP * ((rows + slab_rows - 1) / slab_rows) * 4;
}

int sftg_raster_bands(void) { return RASTER_BANDS; }

/* Resolve CTAs per tile for a launch over `tiles` tiles in all: the knob's number, halved down to 4
 * while the launch would exceed 4096 CTAs, about 7 waves of the 152 SMs x 4 resident ones.  Fewer
 * tiles want the 16 (skinned 320x180 2x, 15 tiles: 0.063 ms against 0.115 with 8; static 640x360 1x, 60
 * tiles: 0.014 against 0.018; atrium 1279x719 1x, 240 tiles: 0.098 against 0.100); with more, a CTA's
 * light list and proxy cache should serve more blocks (1080p, 510 tiles: 0.150 ms with 8, 0.186 with 16
 * at 2x, 0.309 and 0.321 at 4x).  Below 4 the tail grows (1080p 2x 0.184 ms with 2), except where the
 * tiles alone are many waves: 48 views, 16000 tiles: 6.39 ms with 2, 6.54 with 4, 6.86 with 8, 7.77 with 16. */
int sftg_resolve_split(int knob, uint32_t tiles) {
    while (knob > 4 && (uint64_t)tiles * (uint32_t)knob > 4096u) knob /= 2;
    return knob == 4 && tiles > 4096u ? 2 : knob;
}

/* Whether a range's light lists and proxy selections are made once per tile (k_tile_lights) or by
 * each of its resolve CTAs: from 128 tiles on, the selections saved outweigh one more launch on the
 * critical path (510 tiles 4x 0.307 against 0.321 ms, 48 views 6.86 against 7.18, both at 8 CTAs per tile;
 * 240 tiles 1x level; 60 tiles 0.016 against 0.013). */
bool sftg_resolve_records(int knob, uint32_t tiles) { return knob == 2 || (knob == 0 && tiles >= 128u); }

cudaError_t sftg_tile_configure(int max_dynamic_smem) {
    cudaError_t e = cudaSuccess;
    const int S_[3] = { 1, 2, 4 };
    for (int k = 0; k < 3 && e == cudaSuccess; k++) {
        const int need = (int)raster_smem(S_[k], MIN_SLAB_ROWS);
        const int v = need < max_dynamic_smem ? need : max_dynamic_smem;
        if (S_[k] == 1) e = cudaFuncSetAttribute(k_raster<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
        if (S_[k] == 2) e = cudaFuncSetAttribute(k_raster<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
        if (S_[k] == 4) e = cudaFuncSetAttribute(k_raster<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
        if (e != cudaSuccess) break;
        if (S_[k] == 1) e = cudaFuncSetAttribute(k_raster_queue<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
        if (S_[k] == 2) e = cudaFuncSetAttribute(k_raster_queue<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
        if (S_[k] == 4) e = cudaFuncSetAttribute(k_raster_queue<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
    }
    return e;
}

/* CTAs of a persistent launch: as many as are resident at once on all SMs (at least 1), never more
 * than there are items */
template <class K>
static uint32_t queue_grid(K kernel, int threads, size_t smem, uint32_t n_items) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    const uint64_t g = (uint64_t)(sms > 0 ? sms : 1) * (uint64_t)(per_sm > 0 ? per_sm : 1);
    return (uint32_t)(g < n_items ? g : n_items);
}

void sftg_launch_raster(int S, uint32_t tiles, int slab_rows, int bands, uint32_t* queue, cudaStream_t st, const sftg_tile_args& A) {
    if (!tiles) return;
    const size_t sm = raster_smem(S, slab_rows);
    const uint32_t items = sftg_raster_items_max(S, tiles, bands);
    if (queue) {
        if (S == 1) k_raster_queue<1><<<queue_grid(k_raster_queue<1>, RASTER_THREADS, sm, items), RASTER_THREADS, sm, st>>>(A, slab_rows, queue);
        else if (S == 2) k_raster_queue<2><<<queue_grid(k_raster_queue<2>, RASTER_THREADS, sm, items), RASTER_THREADS, sm, st>>>(A, slab_rows, queue);
        else k_raster_queue<4><<<queue_grid(k_raster_queue<4>, RASTER_THREADS, sm, items), RASTER_THREADS, sm, st>>>(A, slab_rows, queue);
        return;
    }
    if (S == 1) k_raster<1><<<items, RASTER_THREADS, sm, st>>>(A, slab_rows);
    else if (S == 2) k_raster<2><<<items, RASTER_THREADS, sm, st>>>(A, slab_rows);
    else k_raster<4><<<items, RASTER_THREADS, sm, st>>>(A, slab_rows);
}

void sftg_launch_tile_lights(uint32_t tile0, uint32_t tiles, cudaStream_t st, const sftg_tile_args& A) {
    if (tiles) k_tile_lights<<<tiles, TILE_THREADS, 0, st>>>(A, tile0);
}

void sftg_launch_resolve(int S, uint32_t tile0, uint32_t tiles, int split, bool records, uint32_t* queue, cudaStream_t st,
                         const sftg_tile_args& A) {
    if (!tiles) return;
    const uint32_t items = tiles * (uint32_t)split;
    if (queue) {
        if (S == 1) k_resolve_queue<1><<<queue_grid(k_resolve_queue<1>, TILE_THREADS, 0, items), TILE_THREADS, 0, st>>>(A, tile0, split, records, items, queue);
        else if (S == 2) k_resolve_queue<2><<<queue_grid(k_resolve_queue<2>, TILE_THREADS, 0, items), TILE_THREADS, 0, st>>>(A, tile0, split, records, items, queue);
        else k_resolve_queue<4><<<queue_grid(k_resolve_queue<4>, TILE_THREADS, 0, items), TILE_THREADS, 0, st>>>(A, tile0, split, records, items, queue);
        return;
    }
    if (S == 1) k_resolve<1><<<items, TILE_THREADS, 0, st>>>(A, tile0, split, records);
    else if (S == 2) k_resolve<2><<<items, TILE_THREADS, 0, st>>>(A, tile0, split, records);
    else k_resolve<4><<<items, TILE_THREADS, 0, st>>>(A, tile0, split, records);
}
