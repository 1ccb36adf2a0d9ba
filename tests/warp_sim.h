/* A warp on the CPU, to run device code that is plain C++ but for its warp collectives: 32 lanes as
 * fibers, each running to its next collective; a collective is carried out once all lanes have come to
 * it.  Lanes that meet different ones, or a lane that ended before, are an error here (on a GPU they wait
 * for one another without end), and so is a warp that takes too many rounds. */
#pragma once
#include <ucontext.h>
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>

#define __global__
#define __device__
#define __forceinline__ inline
#define __restrict__
#define __launch_bounds__(...)
#define __shared__ static
using std::max;
using std::min;
struct sim_dim { unsigned x; };
static sim_dim threadIdx, blockIdx, blockDim;
struct alignas(16) float4 { float x, y, z, w; };
static inline float4 make_float4(float a, float b, float c, float d) { return { a, b, c, d }; }
static inline uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static inline float __uint_as_float(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __fsqrt_rn(float a) { return sqrtf(a); }
static inline int __popc(uint32_t v) { return __builtin_popcount(v); }
static inline int __ffs(uint32_t v) { return __builtin_ffs((int)v); }
static inline uint32_t atomicAdd(uint32_t* p, uint32_t v) { const uint32_t o = *p; *p += v; return o; }

static ucontext_t sim_main, sim_lane[32];
static char* sim_stack[32];
static std::function<void()> sim_fn;
static int sim_cur, sim_site[32];      /* the running lane; where each one waits, 0 once it has ended */
static uint64_t sim_val[2][32];        /* alternating: a lane may be a collective ahead of the others' reads */
static unsigned sim_count[32];

static uint64_t* sim_collect(int site, uint64_t v) {
    const int me = sim_cur;
    uint64_t* const vals = sim_val[sim_count[me]++ & 1];
    vals[me] = v;
    sim_site[me] = site;
    swapcontext(&sim_lane[me], &sim_main);
    return vals;
}
static uint32_t sim_ballot(int site, bool p) {
    const uint64_t* v = sim_collect(site, p);
    uint32_t m = 0;
    for (int l = 0; l < 32; l++) m |= (uint32_t)(v[l] & 1) << l;
    return m;
}
template <class T> static T sim_shfl(int site, T x, int src) {
    uint64_t u = 0;
    memcpy(&u, &x, sizeof(T));
    const uint64_t* v = sim_collect(site, u);
    T r;
    memcpy(&r, &v[src & 31], sizeof(T));
    return r;
}
#define SIM_SITE (__COUNTER__ + 1)     /* two collectives of one line are two */
#define __ballot_sync(mask, p) sim_ballot(SIM_SITE, (p))
#define __any_sync(mask, p) (sim_ballot(SIM_SITE, (p)) != 0)
#define __shfl_sync(mask, v, src) sim_shfl(SIM_SITE, (v), (src))
#define __syncwarp() sim_collect(SIM_SITE, 0)

static void sim_entry() {
    sim_fn();
    sim_site[sim_cur] = 0;
    swapcontext(&sim_lane[sim_cur], &sim_main);
}

/* Runs `kernel` as warp `warp` of block `block`; null when it ended, else what went wrong. */
static const char* sim_warp(unsigned block, unsigned warp, long most, const std::function<void()>& kernel) {
    sim_fn = kernel;
    blockIdx.x = block;
    for (int l = 0; l < 32; l++) {
        if (!sim_stack[l]) sim_stack[l] = (char*)malloc(1 << 17);
        getcontext(&sim_lane[l]);
        sim_lane[l].uc_stack.ss_sp = sim_stack[l];
        sim_lane[l].uc_stack.ss_size = 1 << 17;
        sim_lane[l].uc_link = nullptr;
        makecontext(&sim_lane[l], sim_entry, 0);
        sim_count[l] = 0;
    }
    for (long round = 0; round < most; round++) {
        for (int l = 0; l < 32; l++) {
            sim_cur = l;
            threadIdx.x = warp * 32 + (unsigned)l;
            swapcontext(&sim_main, &sim_lane[l]);
        }
        for (int l = 1; l < 32; l++)
            if (sim_site[l] != sim_site[0]) return "lanes at different collectives";
        if (!sim_site[0]) return nullptr;
    }
    return "no end";
}
