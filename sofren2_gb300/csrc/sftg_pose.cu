/*
 * Skeletal pose evaluation (sft_pose_update, sofren2.c:8952-9108), `per` requests per CTA.
 *
 *   locals     a thread per (request, bone): the bone's T, R and S samplers (the upload keeps, per
 *              animation, the last channel of each node and path, which is the one that wins in
 *              the reference's sequential loop); the keyframe pair by the reference's binary
 *              search, lerp for T and S, sft_q_slerp for R, or the step value; S * (R * T) from
 *              the animated or rest values, else the local bind matrix
 *   hierarchy  four threads per request, one per matrix row, take the bones parents first:
 *              global = local * global[parent], each bone once, as the reference's repeated passes do
 *   posed      inverse bind * global, a thread per (request, bone, row): both outputs leave as
 *              16-byte rows, consecutive over the warp
 * Matrix products follow sft_m_mul (sofren2.c:1668): left-to-right sums of plain products.
 *
 * Half of the issue slots are used, most of them for the slerps and the local products, with 23 of 32
 * threads (bones with and without a rotation sampler share a warp); the waits are for the samplers' keys
 * and at the two barriers (a quarter of the time is the 2.8 KB of matrices a request of 22 bones
 * writes, at the copy rate).  One warp per request, lanes
 * on channels and whole matrices stored per lane, took 361 us for 65536 requests of 22 bones: the
 * hierarchy ran level by level with a few lanes, and each store touched 32 lines.  Now 105 us; 1024
 * requests 14.4 -> 12.4 us.
 */
#include "sftg_types.h"
#include "sftg_kernels.h"

#define POSE_THREADS 128
#define POSE_MAX_PER 32           /* requests per CTA: POSE_THREADS / 4 rows */

__device__ __forceinline__ void mmul(const float* a, const float* b, float* r) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            r[i * 4 + j] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a[i * 4 + 0], b[0 * 4 + j]), __fmul_rn(a[i * 4 + 1], b[1 * 4 + j])),
                                              __fmul_rn(a[i * 4 + 2], b[2 * 4 + j])), __fmul_rn(a[i * 4 + 3], b[3 * 4 + j]));
}

__device__ __forceinline__ void qnorm(float* q) {   /* sft_q_norm */
    const float l2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
    if (l2 != 0.f) { const float il = __fdiv_rn(1.f, __fsqrt_rn(l2)); q[0] *= il; q[1] *= il; q[2] *= il; q[3] *= il; }
}

__device__ void slerp(const float* a, const float* b_in, float t, float* out) {   /* sft_q_slerp (1857-1892) */
    float b[4] = { b_in[0], b_in[1], b_in[2], b_in[3] };
    float dot = a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3];
    if (dot < 0.f) { b[0] = -b[0]; b[1] = -b[1]; b[2] = -b[2]; b[3] = -b[3]; dot = -dot; }
    if (dot > 0.9995f) {
#pragma unroll
        for (int k = 0; k < 4; k++) out[k] = a[k] + t * (b[k] - a[k]);
        qnorm(out);
        return;
    }
    const float th0 = acosf(dot), th = th0 * t, st = sinf(th), is0 = __fdiv_rn(1.f, sinf(th0));
    const float s0 = cosf(th) - dot * st * is0, s1 = st * is0;
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = a[k] * s0 + b[k] * s1;
    qnorm(out);
}

__device__ void from_quat(const float* q, float* m) {   /* sft_m_from_quat (1822-1850) */
    const float x2 = q[0] + q[0], y2 = q[1] + q[1], z2 = q[2] + q[2];
    const float xx = q[0] * x2, xy = q[0] * y2, xz = q[0] * z2, yy = q[1] * y2, yz = q[1] * z2, zz = q[2] * z2;
    const float wx = q[3] * x2, wy = q[3] * y2, wz = q[3] * z2;
    m[0] = 1.f - (yy + zz); m[1] = xy + wz; m[2] = xz - wy; m[3] = 0.f;
    m[4] = xy - wz; m[5] = 1.f - (xx + zz); m[6] = yz + wx; m[7] = 0.f;
    m[8] = xz + wy; m[9] = yz - wx; m[10] = 1.f - (xx + yy); m[11] = 0.f;
    m[12] = 0.f; m[13] = 0.f; m[14] = 0.f; m[15] = 1.f;
}

/* A sampler at `time`: xyz (path T or S) or the slerped quaternion (R) into val. */
__device__ void sample(const sftg_pose_tables& T, int sampler, bool rotation, float time, float* val) {
    const sftg_sampler_dev sm = T.samplers[sampler];
    const float* in = T.keys + sm.input_base;
    const float* out = T.keys + sm.output_base;
    int f0 = 0, f1 = 0;
    float t = 0.f;
    if (time <= in[0]) {
        f0 = f1 = 0;
    } else if (time >= in[sm.count - 1]) {
        f0 = f1 = sm.count - 1;
    } else {
        int low = 0, high = sm.count - 1;
        while (low <= high) {
            const int mid = low + (high - low) / 2;
            if (time < in[mid]) high = mid - 1;
            else if (time >= in[mid + 1]) low = mid + 1;
            else { f0 = mid; f1 = mid + 1; break; }
        }
        const float dt = in[f1] - in[f0];
        t = (dt > 0.0001f) ? __fdiv_rn(time - in[f0], dt) : 0.f;
    }
    if (rotation) {
        if (sm.is_step) { for (int q = 0; q < 4; q++) val[q] = out[f0 * 4 + q]; }
        else slerp(out + f0 * 4, out + f1 * 4, t, val);
    } else {
        for (int q = 0; q < 3; q++) {
            const float v0 = out[f0 * 4 + q], v1 = out[f1 * 4 + q];
            val[q] = sm.is_step ? v0 : v0 + (v1 - v0) * t;
        }
    }
}

/* row * m for a row and the four rows of a matrix, in mmul's order */
__device__ __forceinline__ float4 row_mul(float4 a, const float4* m) {
    const float4 m0 = m[0], m1 = m[1], m2 = m[2], m3 = m[3];
#define COL(c) __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a.x, m0.c), __fmul_rn(a.y, m1.c)), __fmul_rn(a.z, m2.c)), __fmul_rn(a.w, m3.c))
    return make_float4(COL(x), COL(y), COL(z), COL(w));
#undef COL
}

/* VEC: the output arrays are 16-byte aligned */
template <bool VEC>
__device__ __forceinline__ void store_row(float* p, float4 v) {
    if (VEC) *(float4*)p = v;
    else { p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w; }
}

template <bool VEC>
__global__ void __launch_bounds__(POSE_THREADS)
k_pose(const sftg_pose_tables T, const sftg_pose_request* __restrict__ reqs, const uint32_t* __restrict__ out_off, uint32_t n, int per,
       int stride, float* __restrict__ posed, float* __restrict__ global_out)
{
    extern __shared__ float4 s_g[];   /* [per][stride][4 rows]: local, then global matrices; stride is odd (banks) */
    __shared__ int s_nb[POSE_MAX_PER];
    __shared__ uint32_t s_bone[POSE_MAX_PER], s_win[POSE_MAX_PER], s_order[POSE_MAX_PER], s_off[POSE_MAX_PER];
    __shared__ float s_time[POSE_MAX_PER];
    const int tid = threadIdx.x;
    if (tid < per) {
        const uint32_t k = blockIdx.x * (uint32_t)per + tid;
        int nb = 0;   /* 0: a request that leaves its matrices untouched */
        if (k < n) {
            const sftg_pose_request R = reqs[k];
            if (R.skeleton >= 0 && (uint32_t)R.skeleton < T.n_skels) {
                const sftg_skel_dev sk = T.skels[R.skeleton];
                if (R.animation >= 0 && R.animation < (int)sk.anim_count) {   /* else sft_pose_update returns early */
                    const sftg_anim_dev an = T.anims[sk.anim_base + R.animation];
                    nb = (int)sk.bone_count;
                    s_bone[tid] = sk.bone_base; s_order[tid] = sk.order_base; s_win[tid] = an.win_base;
                    s_off[tid] = out_off[k];
                    s_time[tid] = an.duration > 1e-6f ? fmodf(R.time, an.duration) : R.time;
                }
            }
        }
        s_nb[tid] = nb;
    }
    __syncthreads();
    /* local matrices */
    for (int i = tid; i < per * stride; i += POSE_THREADS) {
        const int r = i / stride, b = i - r * stride;
        if (b >= s_nb[r]) continue;
        const sftg_bone_dev& bd = T.bones[s_bone[r] + b];
        const int* win = T.wins + (size_t)s_win[r] + 3 * b;
        const int wt = win[0], wr = win[1], ws = win[2];
        float4* g = s_g + 4 * (size_t)i;
        if (wt >= 0 || wr >= 0 || ws >= 0) {
            float tp[4] = { bd.base_t[0], bd.base_t[1], bd.base_t[2], 0.f };
            float rq[4] = { bd.base_r[0], bd.base_r[1], bd.base_r[2], bd.base_r[3] };
            float sc[4] = { bd.base_s[0], bd.base_s[1], bd.base_s[2], 0.f };
            const float time = s_time[r];
            if (wr >= 0) sample(T, wr, true, time, rq);
            if (wt >= 0) sample(T, wt, false, time, tp);
            if (ws >= 0) sample(T, ws, false, time, sc);
            float Tm[16] = { 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, tp[0], tp[1], tp[2], 1 };
            float Sm[16] = { sc[0], 0, 0, 0, 0, sc[1], 0, 0, 0, 0, sc[2], 0, 0, 0, 0, 1 };
            float Rm[16], RT[16], L[16];
            from_quat(rq, Rm);
            mmul(Rm, Tm, RT);
            mmul(Sm, RT, L);
#pragma unroll
            for (int q = 0; q < 4; q++) g[q] = make_float4(L[4 * q], L[4 * q + 1], L[4 * q + 2], L[4 * q + 3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) g[q] = ((const float4*)bd.local_bind)[q];
        }
    }
    __syncthreads();
    /* hierarchy: the order table holds bone | parent << 16 (0xFFFF: none), parents first */
    if (tid < ((per * 4 + 31) & ~31)) {   /* whole warps */
        const int r = tid >> 2, row = tid & 3;
        const int nb = r < per ? s_nb[r] : 0;   /* per may be 1 or 2 */
        const uint32_t* order = T.order + (nb ? s_order[r] : 0u);
        float4* g = s_g + (size_t)r * stride * 4;
        const int steps = __reduce_max_sync(0xFFFFFFFFu, nb);
        uint32_t next = nb ? order[0] : 0u;
        for (int q = 0; q < steps; q++) {
            const uint32_t e = next;
            if (q + 1 < nb) next = order[q + 1];
            if (q < nb && (e >> 16) != 0xFFFFu) {
                const int b = (int)(e & 0xFFFFu), p = (int)(e >> 16);
                g[b * 4 + row] = row_mul(g[b * 4 + row], g + p * 4);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    /* posed = inverse bind * global */
    for (int i = tid; i < per * stride * 4; i += POSE_THREADS) {
        const int m = i >> 2, row = i & 3, r = m / stride, b = m - r * stride;
        if (b >= s_nb[r]) continue;
        const float4 iv = ((const float4*)T.bones[s_bone[r] + b].inverse_bind)[row];
        const size_t o = ((size_t)s_off[r] + b) * 16 + 4 * row;
        store_row<VEC>(posed + o, row_mul(iv, s_g + 4 * (size_t)m));
        if (global_out) store_row<VEC>(global_out + o, s_g[i]);
    }
}

void sftg_launch_pose(const sftg_pose_tables& T, const sftg_pose_request* reqs, const uint32_t* out_off, uint32_t n, float* posed,
                      float* global, cudaStream_t st) {
    if (!n) return;
    /* requests per CTA: as many as 24 KB of matrices hold (22 bones: 16; 65536 requests 105 us, with 48 KB
     * 141, 16384 requests 33 us, with 12 KB 37), fewer while that leaves SMs without two CTAs */
    const int stride = (int)(T.max_bones | 1u);
    int per = POSE_MAX_PER;
    while (per > 1 && ((size_t)per * stride * 64 > 24u * 1024u || (uint64_t)per * 304u > n)) per /= 2;
    const size_t sm = (size_t)per * stride * 64;
    const uint32_t grid = (n + per - 1) / per;
    if ((((uintptr_t)posed | (uintptr_t)global) & 15u) == 0) k_pose<true><<<grid, POSE_THREADS, sm, st>>>(T, reqs, out_off, n, per, stride, posed, global);
    else k_pose<false><<<grid, POSE_THREADS, sm, st>>>(T, reqs, out_off, n, per, stride, posed, global);
}
