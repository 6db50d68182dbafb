// attn_fused.cu — one-launch decode attention of the chain lane: rope(q), rope(k) -> K cache,
// v -> V cache, GQA split-K attention and the merge of the splits.
//
// The reference runs this as five dispatches (tensormark/metal.h:3950-3967 rope_q, 3968-4005
// rope_k_cache, 4006-4030 v_cache, 2739-2859 / 4153-4222 attention and its split merge). On a GPU
// whose GEMVs take a few microseconds each, five launches with a dependent chain of cache misses
// behind each cost more than the attention itself, so the chain form does it in one kernel:
//
//   grid (KVH, nsplit), 4 warps. The positions [0, pos] are cut into tiles of 32; a CTA owns a
//   contiguous range of tiles of one KV head and its warps take them round-robin.
//   * Every CTA rotates the REP query heads of its KV head into shared memory (q is tiny).
//   * The CTA whose range holds position `pos` rotates the new k, stores k and v into the caches
//     and takes its own scores and values of that row from shared memory.
//   * Scores: one LANE per POSITION. A lane reads its own K row (contiguous) and dots it with the
//     query heads from shared memory (broadcast reads): no shuffle per position, 32 independent
//     row reads in flight per warp.
//   * Values: one lane per dh/32 DIMS. For each position of the tile the lanes read one V row
//     (coalesced) and the position's weights come by shuffle.
//   * A CTA leaves an unnormalised partial (max, sum, acc) per head; the CTA that arrives last at a
//     KV head's counter merges the nsplit partials and writes the output rows.
//
// The arithmetic is the reference's (fp32 scores, exp of score - max, value sum, one division);
// only the order of the sums differs, so results agree with the oracle to rounding.
#include "common.cuh"
#include "glue.h"

#include <cstdlib>

#include <cuda_fp16.h>
#include <math_constants.h>

namespace tmc {

namespace {

constexpr unsigned kMaxSplits = 32;      // a lane each in the merge

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// The rotation, with its contractions written out: what a token's K row is must not depend on how a compiler places them.
__device__ __forceinline__ float rope_lo(float a, float b, float2 cs) { return fmaf(a, cs.x, -__fmul_rn(b, cs.y)); }
__device__ __forceinline__ float rope_hi(float a, float b, float2 cs) { return fmaf(a, cs.y, __fmul_rn(b, cs.x)); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <typename T> __device__ __forceinline__ T to_cache(float v);
template <> __device__ __forceinline__ float to_cache<float>(float v) { return v; }
template <> __device__ __forceinline__ __half to_cache<__half>(float v) { return __float2half_rn(v); }

// Raw loads are issued in batches before anything is computed on them: the kernel is a chain of
// cache-miss latencies, so what matters is how many loads are in flight, not how many are issued.
template <typename T> struct Raw8;
template <> struct Raw8<__half> { uint4 u; };
template <> struct Raw8<float> { float4 a, b; };
__device__ __forceinline__ void fetch8(const __half* p, Raw8<__half>& r) { r.u = __ldcg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ void fetch8(const float* p, Raw8<float>& r) {
    r.a = __ldcg(reinterpret_cast<const float4*>(p)); r.b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
}
__device__ __forceinline__ void unpack8(const Raw8<__half>& r, float (&f)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&r.u);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 t = __half22float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ void unpack8(const Raw8<float>& r, float (&f)[8]) {
    f[0] = r.a.x; f[1] = r.a.y; f[2] = r.a.z; f[3] = r.a.w; f[4] = r.b.x; f[5] = r.b.y; f[6] = r.b.z; f[7] = r.b.w;
}
// DPL consecutive cache elements (DPL = 2 or 4): raw fetch now, floats later.
template <typename T, int DPL> struct RawV;
template <> struct RawV<__half, 4> { uint2 u; };
template <> struct RawV<__half, 2> { unsigned u; };
template <> struct RawV<float, 4> { float4 u; };
template <> struct RawV<float, 2> { float2 u; };
__device__ __forceinline__ void fetchv(const __half* p, RawV<__half, 4>& r) { r.u = __ldcg(reinterpret_cast<const uint2*>(p)); }
__device__ __forceinline__ void fetchv(const __half* p, RawV<__half, 2>& r) { r.u = __ldcg(reinterpret_cast<const unsigned*>(p)); }
__device__ __forceinline__ void fetchv(const float* p, RawV<float, 4>& r) { r.u = __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void fetchv(const float* p, RawV<float, 2>& r) { r.u = __ldcg(reinterpret_cast<const float2*>(p)); }
__device__ __forceinline__ void unpackv(const RawV<__half, 4>& r, float (&f)[4]) {
    const __half2* h = reinterpret_cast<const __half2*>(&r.u);
    const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
__device__ __forceinline__ void unpackv(const RawV<__half, 2>& r, float (&f)[2]) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r.u));
    f[0] = a.x; f[1] = a.y;
}
__device__ __forceinline__ void unpackv(const RawV<float, 4>& r, float (&f)[4]) { f[0] = r.u.x; f[1] = r.u.y; f[2] = r.u.z; f[3] = r.u.w; }
__device__ __forceinline__ void unpackv(const RawV<float, 2>& r, float (&f)[2]) { f[0] = r.u.x; f[1] = r.u.y; }

// A warp's part of a split: `tile`, `tile` + 4, ... below t1, for the REP query heads. kn, vn: the new position's rows
// (the cache's rows of it may not be visible yet when the first tile is fetched).
template <typename T, int DPL, int REP> struct Tile {
    static constexpr int dh = DPL * 32;
    Raw8<T> raw[dh / 8];
    RawV<T, DPL> vraw[32];                                     // rows past the tile's last position repeat it, their weight is 0
    __device__ __forceinline__ void fetch(const T* kbase, const T* vbase, uint32_t t, uint32_t allow, uint32_t lane) {   // this lane's K row (lane = position) and its dims of the 32 V rows
        const uint32_t p = t * 32 + lane, np = min(32u, allow - t * 32);
        const T* krow = kbase + (size_t)min(p, allow - 1) * dh;
        const T* vrow = vbase + (size_t)t * 32 * dh + lane * DPL;
#pragma unroll
        for (int c = 0; c < dh / 8; ++c) fetch8(krow + c * 8, raw[c]);
#pragma unroll
        for (int k = 0; k < 32; ++k) fetchv(vrow + (size_t)min((uint32_t)k, np - 1) * dh, vraw[k]);
    }
    // what aliases the new position's row, taken from shared memory
    __device__ __forceinline__ void patch(const T* kn, const T* vn, uint32_t kpos, uint32_t lane) {
        if (lane >= kpos) {
#pragma unroll
            for (int c = 0; c < dh / 8; ++c) raw[c] = *reinterpret_cast<const Raw8<T>*>(kn + c * 8);
        }
        const RawV<T, DPL> v = *reinterpret_cast<const RawV<T, DPL>*>(vn + lane * DPL);
#pragma unroll
        for (int k = 0; k < 32; ++k)
            if ((uint32_t)k >= kpos) vraw[k] = v;
    }
    __device__ __forceinline__ void attend(const T* kbase, const T* vbase, const T* kn, const T* vn, uint32_t tile, uint32_t t1, uint32_t tiles,
                                           uint32_t allow, uint32_t lane, const float (*qs)[dh], float* sm_m, float* sm_l, float (*sm_acc)[dh]) {
        float m[REP], l[REP], acc[REP][DPL];
#pragma unroll
        for (int r = 0; r < REP; ++r) {
            m[r] = -CUDART_INF_F; l[r] = 0.f;
#pragma unroll
            for (int d = 0; d < DPL; ++d) acc[r][d] = 0.f;
        }
        for (uint32_t t = tile; t < t1; t += 4) {
            const uint32_t p = t * 32 + lane;
            const bool live = p < allow;
            float s[REP];
#pragma unroll
            for (int r = 0; r < REP; ++r) s[r] = 0.f;
            // Every load of a tile is requested before anything is computed on it; the first tile's were before the wait.
            if (t != tile) fetch(kbase, vbase, t, allow, lane);
            if (t == tiles - 1) patch(kn, vn, allow - 1 - t * 32, lane);
            if (live) {
#pragma unroll
                for (int c = 0; c < dh / 8; ++c) {
                    float kf[8];
                    unpack8(raw[c], kf);
#pragma unroll
                    for (int r = 0; r < REP; ++r) {
                        const float4 qa = *reinterpret_cast<const float4*>(&qs[r][c * 8]);
                        const float4 qb = *reinterpret_cast<const float4*>(&qs[r][c * 8 + 4]);
                        float v = s[r];
                        v = fmaf(qa.x, kf[0], v); v = fmaf(qa.y, kf[1], v); v = fmaf(qa.z, kf[2], v); v = fmaf(qa.w, kf[3], v);
                        v = fmaf(qb.x, kf[4], v); v = fmaf(qb.y, kf[5], v); v = fmaf(qb.z, kf[6], v); v = fmaf(qb.w, kf[7], v);
                        s[r] = v;
                    }
                }
            }
            // tile softmax statistics and this lane's weight per head
            float pw[REP];
#pragma unroll
            for (int r = 0; r < REP; ++r) {
                float tm = live ? s[r] : -CUDART_INF_F;
#pragma unroll
                for (int o = 16; o; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
                const float mn = fmaxf(m[r], tm);                 // finite: every tile holds at least one live position
                const float corr = __expf(m[r] - mn);
                pw[r] = live ? __expf(s[r] - mn) : 0.f;
                float ts = pw[r];
#pragma unroll
                for (int o = 16; o; o >>= 1) ts += __shfl_xor_sync(0xffffffffu, ts, o);
                l[r] = l[r] * corr + ts;
#pragma unroll
                for (int d = 0; d < DPL; ++d) acc[r][d] *= corr;
                m[r] = mn;
            }
            // values: lanes own dims, the tile's positions one after another (weight 0 past the last position)
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                float vf[DPL];
                unpackv(vraw[k], vf);
#pragma unroll
                for (int r = 0; r < REP; ++r) {
                    const float w = __shfl_sync(0xffffffffu, pw[r], k);
#pragma unroll
                    for (int d = 0; d < DPL; ++d) acc[r][d] = fmaf(w, vf[d], acc[r][d]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < REP; ++r) {
            if (lane == 0) { sm_m[r] = m[r]; sm_l[r] = l[r]; }
#pragma unroll
            for (int d = 0; d < DPL; ++d) sm_acc[r][lane * DPL + d] = acc[r][d];
        }
    }
};

// The same for one tile that lies in shared memory and NH of the query heads: what a warp's first tile comes to in attend(),
// operation for operation. kt: rows of KST halves, vt: rows of dh.
template <int DPL, int NH, int KST>
__device__ __forceinline__ void attend_shared(const __half* kt, const __half* vt, bool live, uint32_t lane, const float (*qs)[DPL * 32], float* sm_m, float* sm_l,
                                              float (*sm_acc)[DPL * 32]) {
    constexpr int dh = DPL * 32;
    float s[NH], pw[NH], acc[NH][DPL];
#pragma unroll
    for (int r = 0; r < NH; ++r) {
        s[r] = 0.f;
#pragma unroll
        for (int d = 0; d < DPL; ++d) acc[r][d] = 0.f;
    }
#pragma unroll 4
    for (int c = 0; c < dh / 8; ++c) {
        Raw8<__half> raw;
        raw.u = *reinterpret_cast<const uint4*>(kt + lane * KST + c * 8);
        float kf[8];
        unpack8(raw, kf);
#pragma unroll
        for (int r = 0; r < NH; ++r) {
            const float4 qa = *reinterpret_cast<const float4*>(&qs[r][c * 8]);
            const float4 qb = *reinterpret_cast<const float4*>(&qs[r][c * 8 + 4]);
            float v = s[r];
            v = fmaf(qa.x, kf[0], v); v = fmaf(qa.y, kf[1], v); v = fmaf(qa.z, kf[2], v); v = fmaf(qa.w, kf[3], v);
            v = fmaf(qb.x, kf[4], v); v = fmaf(qb.y, kf[5], v); v = fmaf(qb.z, kf[6], v); v = fmaf(qb.w, kf[7], v);
            s[r] = v;
        }
    }
#pragma unroll
    for (int r = 0; r < NH; ++r) {
        float tm = live ? s[r] : -CUDART_INF_F;
#pragma unroll
        for (int o = 16; o; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
        pw[r] = live ? __expf(s[r] - tm) : 0.f;
        float ts = pw[r];
#pragma unroll
        for (int o = 16; o; o >>= 1) ts += __shfl_xor_sync(0xffffffffu, ts, o);
        if (lane == 0) { sm_m[r] = tm; sm_l[r] = ts; }
    }
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
        const RawV<__half, DPL> raw = *reinterpret_cast<const RawV<__half, DPL>*>(vt + k * dh + lane * DPL);
        float vf[DPL];
        unpackv(raw, vf);
#pragma unroll
        for (int r = 0; r < NH; ++r) {
            const float w = __shfl_sync(0xffffffffu, pw[r], k);
#pragma unroll
            for (int d = 0; d < DPL; ++d) acc[r][d] = fmaf(w, vf[d], acc[r][d]);
        }
    }
#pragma unroll
    for (int r = 0; r < NH; ++r)
#pragma unroll
        for (int d = 0; d < DPL; ++d) sm_acc[r][lane * DPL + d] = acc[r][d];
}

template <typename T, int DPL, int REP>
__global__ void __launch_bounds__(128) attn_fused_kernel(const float* qkv, T* kc, T* vc, float* part, float* stat,
                                                          unsigned* counters, float* out, uint32_t H, uint32_t KVH,
                                                          uint32_t ctx, float scale, const float2* __restrict__ tbl,
                                                          uint32_t tbl_n, const int* st, unsigned long long* trace) {
    unsigned long long* tr = nullptr;                         // timeline of CTA (0, 0), thread 0 (see tm_cuda_trace_read)
    if (trace && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        const unsigned long long slot = atomicAdd(trace, 1ull);
        if (slot < (unsigned long long)kTraceLaunches) { tr = trace + 1 + slot * kTraceWords; tr[0] = now_ns(); }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr int dh = DPL * 32, half = dh / 2;
    const uint32_t kv = blockIdx.x, split = blockIdx.y, nsplit = gridDim.y;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The position was written by the previous token's last kernel and the cache rows below it by earlier tokens:
    // both are safe to read before this token's q|k|v GEMV has finished, and this CTA is resident (and idle) for
    // several microseconds before that. So the first tile's loads, with their page walks and DRAM latency, are
    // requested now; only the row of the new position is put in after the wait.
    const int pos_i = *(volatile const int*)st;
    const bool valid = !(pos_i < 0 || (uint32_t)pos_i >= ctx || (uint32_t)pos_i * half + half > tbl_n);   // same guard as the separate kernels
    const uint32_t pos = valid ? (uint32_t)pos_i : 0u, allow = pos + 1;
    const uint32_t tiles = (allow + 31) / 32, tps = (tiles + nsplit - 1) / nsplit;
    const uint32_t t0 = min(tiles, split * tps), t1 = min(tiles, t0 + tps), used = (tiles + tps - 1) / tps;    // used: splits that have a tile
    const T* kbase = kc + (size_t)kv * ctx * dh;
    const T* vbase = vc + (size_t)kv * ctx * dh;
    // Splits of one or two tiles (an 8-head fp16 cache: up to 1216 positions) take their tiles through shared memory, and the
    // warps share the query heads out between them: with a tile per warp three of the four had nothing to do and the fourth
    // was a chain of REP * 64 dependent steps. Longer splits have a tile for every warp.
    constexpr int MAXT = sizeof(T) != 2 ? 0 : REP == 8 && DPL == 4 ? 1 : 2, KST = dh + 8;
    constexpr int NH = REP < 4 ? 1 : REP / 4, GROUPS = REP / NH;
    __shared__ __align__(16) T kt[MAXT ? MAXT : 1][MAXT ? 32 : 1][KST];
    __shared__ __align__(16) T vt[MAXT ? MAXT : 1][MAXT ? 32 : 1][dh];
    const bool shared = tps <= (uint32_t)MAXT;
    const uint32_t t_first = t0 + warp;
    Tile<T, DPL, REP> tile;
    if (valid && shared) {
        constexpr uint32_t C = dh / 8;                         // 16-byte pieces of a row
        for (uint32_t i = threadIdx.x; i < (t1 - t0) * 32u * C; i += 128) {
            const uint32_t t = i / (32u * C), r = i / C % 32u, c = i % C, p = (t0 + t) * 32u + r;
            T *kd = &kt[MAXT ? t : 0][MAXT ? r : 0][8 * c], *vd = &vt[MAXT ? t : 0][MAXT ? r : 0][8 * c];
            if (p < pos) {
                cp_async16(kd, kbase + (size_t)p * dh + 8 * c);
                cp_async16(vd, vbase + (size_t)p * dh + 8 * c);
            } else if (p > pos) {
                *reinterpret_cast<uint4*>(kd) = make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(vd) = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    } else if (valid && t_first < t1) {
        tile.fetch(kbase, vbase, t_first, allow, lane);
    }
    const float2 cs = valid ? tbl[(size_t)pos * half + threadIdx.x % half] : make_float2(0.f, 0.f);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tr) tr[1] = now_ns();
    if (!valid || t0 >= t1) return;                           // a split without positions leaves nothing to merge

    __shared__ __align__(16) float qs[REP][dh];
    __shared__ __align__(16) T knew[dh];
    __shared__ __align__(16) T vnew[dh];
    __shared__ __align__(16) float sm_acc[4][REP][dh];
    __shared__ float sm_m[4][REP], sm_l[4][REP];
    __shared__ float cm[REP][kMaxSplits], inv_l[REP];
    __shared__ int sm_last;

    // ---- rope(q) for this KV head's query heads, scaled, into shared memory; the new position's k (rotated) and v into
    // the caches and into shared memory, by the CTA that attends it. All loads are requested before the first is used.
    {
        constexpr int NQ = (REP * half + 127) / 128;
        const uint32_t j = threadIdx.x % half;
        const bool newest = t1 == tiles;
        float a[NQ], b[NQ], ka = 0.f, kb = 0.f, va = 0.f;
#pragma unroll
        for (int n = 0; n < NQ; ++n) {
            const uint32_t r = (threadIdx.x + n * 128u) / half;
            if (r < (uint32_t)REP) { const float* q = qkv + (size_t)(kv * REP + r) * dh; a[n] = __ldcg(q + j); b[n] = __ldcg(q + j + half); }
        }
        if (newest && threadIdx.x < half) { const float* kn = qkv + (size_t)(H + kv) * dh; ka = __ldcg(kn + j); kb = __ldcg(kn + j + half); }
        if (newest && threadIdx.x < dh) va = __ldcg(qkv + (size_t)(H + KVH + kv) * dh + threadIdx.x);
#pragma unroll
        for (int n = 0; n < NQ; ++n) {
            const uint32_t r = (threadIdx.x + n * 128u) / half;
            if (r < (uint32_t)REP) {
                qs[r][j] = rope_lo(a[n], b[n], cs) * scale;
                qs[r][j + half] = rope_hi(a[n], b[n], cs) * scale;
            }
        }
        if (newest) {
            T* kdst = kc + ((size_t)kv * ctx + pos) * dh;
            T* vdst = vc + ((size_t)kv * ctx + pos) * dh;
            if (threadIdx.x < half) {
                kdst[j] = knew[j] = to_cache<T>(rope_lo(ka, kb, cs));
                kdst[j + half] = knew[j + half] = to_cache<T>(rope_hi(ka, kb, cs));
            }
            if (threadIdx.x < dh) vdst[threadIdx.x] = vnew[threadIdx.x] = to_cache<T>(va);
            if (shared) {                                      // its row of the tile
                const uint32_t t = MAXT ? tiles - 1 - t0 : 0u, r = MAXT ? pos % 32u : 0u;
                if (threadIdx.x < half) { kt[t][r][j] = knew[j]; kt[t][r][j + half] = knew[j + half]; }
                if (threadIdx.x < dh) vt[t][r][threadIdx.x] = vnew[threadIdx.x];
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (tr) tr[2] = now_ns();

    const uint32_t vwarps = shared ? t1 - t0 : 4u;             // partials of the split
    if constexpr (MAXT != 0) {
        if (shared) {
            for (uint32_t i = warp; i < vwarps * GROUPS; i += 4) {
                const uint32_t t = i / GROUPS, r0 = i % GROUPS * NH;
                attend_shared<DPL, NH, KST>(&kt[t][0][0], &vt[t][0][0], (t0 + t) * 32u + lane < allow, lane, qs + r0, sm_m[t] + r0, sm_l[t] + r0, sm_acc[t] + r0);
            }
        }
    }
    if (!shared) tile.attend(kbase, vbase, knew, vnew, t_first, t1, tiles, allow, lane, qs, sm_m[warp], sm_l[warp], sm_acc[warp]);
    if (tr) tr[4] = now_ns();
    // ---- merge the warps, leave this split's partial. A thread takes four dims of one head, here and below: this part of the
    // kernel runs once, by a few warps, so its time is the latency of its steps and of fetching its code. (Four outputs apart
    // per thread, unrolled over heads and splits, with a fence by every thread: 2.8 us to the counter and 4.5 behind it.)
    __syncthreads();
    constexpr int QUADS = REP * dh / 4, NV = (QUADS + 127) / 128;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const uint32_t q = threadIdx.x + n * 128u, r = q / (dh / 4), d = q % (dh / 4) * 4;
        if (q < (uint32_t)QUADS) {
            float M = -CUDART_INF_F;
#pragma unroll
            for (int w = 0; w < 4; ++w) if (w < (int)vwarps) M = fmaxf(M, sm_m[w][r]);
            float L = 0.f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < 4; ++w)
                if (w < (int)vwarps) {
                    const float f = sm_m[w][r] == -CUDART_INF_F ? 0.f : __expf(sm_m[w][r] - M);
                    const float4 a = *reinterpret_cast<const float4*>(&sm_acc[w][r][d]);
                    L = fmaf(f, sm_l[w][r], L);
                    o.x = fmaf(f, a.x, o.x); o.y = fmaf(f, a.y, o.y); o.z = fmaf(f, a.z, o.z); o.w = fmaf(f, a.w, o.w);
                }
            const size_t head = (size_t)split * H + kv * REP + r;
            *reinterpret_cast<float4*>(part + head * dh + d) = o;
            if (d == 0) *reinterpret_cast<float2*>(stat + head * 2) = make_float2(M, L);
        }
    }

    // ---- the CTA that arrives last at this KV head merges the splits
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned prev;                                        // releases the CTA's partial (the barrier orders it), acquires the others'
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(&counters[kv]) : "memory");
        sm_last = prev == used - 1;
        if (sm_last) counters[kv] = 0u;                       // re-armed for the next launch
    }
    __syncthreads();
    if (tr) { tr[5] = now_ns(); tr[3] = tr[5]; }
    if (!sm_last) return;
    // BATCH splits are requested at a time, the first ones before the weights are known.
    constexpr int BATCH = NV > 1 ? 5 : 10;
    float4 v[NV][BATCH], o[NV];
    auto request = [&](uint32_t s0) {
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const float* from = part + ((size_t)s0 * H + kv * REP) * dh + 4 * (threadIdx.x + n * 128u);
#pragma unroll
            for (int k = 0; k < BATCH; ++k)
                if (s0 + k < used && threadIdx.x + n * 128u < (uint32_t)QUADS) v[n][k] = __ldcg(reinterpret_cast<const float4*>(from + (size_t)k * H * dh));
        }
    };
    request(0);
    // the splits' weights: a warp per head, a lane per split
    for (uint32_t r = warp; r < (uint32_t)REP; r += 4) {
        float2 ml = make_float2(-CUDART_INF_F, 0.f);
        if (lane < used) ml = __ldcg(reinterpret_cast<const float2*>(stat + ((size_t)lane * H + kv * REP + r) * 2));
        float M = ml.x;
#pragma unroll
        for (int sh = 16; sh; sh >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, sh));
        const float wgt = ml.x == -CUDART_INF_F ? 0.f : __expf(ml.x - M);
        float L = 0.f;
        for (uint32_t s2 = 0; s2 < used; ++s2) L = fmaf(__shfl_sync(0xffffffffu, wgt, s2), __shfl_sync(0xffffffffu, ml.y, s2), L);
        cm[r][lane] = wgt;
        if (lane == 0) inv_l[r] = 1.0f / L;
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NV; ++n) o[n] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < used; s0 += BATCH) {
        if (s0) request(s0);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const uint32_t r = min((threadIdx.x + n * 128u) / (dh / 4), (uint32_t)(REP - 1));
#pragma unroll
            for (int k = 0; k < BATCH; ++k)
                if (s0 + k < used) {
                    const float w = cm[r][s0 + k];
                    o[n].x = __fadd_rn(o[n].x, __fmul_rn(w, v[n][k].x)); o[n].y = __fadd_rn(o[n].y, __fmul_rn(w, v[n][k].y));
                    o[n].z = __fadd_rn(o[n].z, __fmul_rn(w, v[n][k].z)); o[n].w = __fadd_rn(o[n].w, __fmul_rn(w, v[n][k].w));
                }
        }
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        const uint32_t q = threadIdx.x + n * 128u;
        if (q < (uint32_t)QUADS) {
            const float w = inv_l[q / (dh / 4)];
            *reinterpret_cast<float4*>(out + (size_t)(kv * REP) * dh + 4 * q) = make_float4(o[n].x * w, o[n].y * w, o[n].z * w, o[n].w * w);
        }
    }
}

unsigned* attn_counters() {
    static unsigned* p = nullptr;
    if (!p) {
        if (cudaMalloc(&p, 1024 * sizeof(unsigned)) != cudaSuccess) { cudaGetLastError(); p = nullptr; return nullptr; }
        cudaMemset(p, 0, 1024 * sizeof(unsigned));
    }
    return p;
}

template <typename T, int DPL, int REP>
void launch_one(dim3 grid, cudaStream_t st, const float* qkv, void* kc, void* vc, float* part, float* stat, unsigned* counters,
                float* out, unsigned H, unsigned KVH, unsigned ctx, float scale, const float* tbl, unsigned tbl_n, const int* state) {
    static const bool pdl = [] { const char* e = std::getenv("TM_GLUE_PDL"); return !(e && *e == '0'); }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(128); cfg.dynamicSmemBytes = 0; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, attn_fused_kernel<T, DPL, REP>, qkv, (T*)kc, (T*)vc, part, stat, counters, out, (uint32_t)H, (uint32_t)KVH,
                       (uint32_t)ctx, scale, (const float2*)tbl, (uint32_t)tbl_n, state, device_trace());
}

template <typename T, int DPL>
bool launch_rep(unsigned REP, dim3 grid, cudaStream_t st, const float* qkv, void* kc, void* vc, float* part, float* stat,
                unsigned* counters, float* out, unsigned H, unsigned KVH, unsigned ctx, float scale, const float* tbl,
                unsigned tbl_n, const int* state) {
    switch (REP) {
        case 1: launch_one<T, DPL, 1>(grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_n, state); return true;
        case 2: launch_one<T, DPL, 2>(grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_n, state); return true;
        case 4: launch_one<T, DPL, 4>(grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_n, state); return true;
        case 8: launch_one<T, DPL, 8>(grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_n, state); return true;
        default: return fail("attention: REP=%u unsupported (1, 2, 4 or 8)", REP);
    }
}

}  // namespace

unsigned attn_fused_splits(unsigned H, unsigned KVH, unsigned dh, unsigned ctx, size_t scratch_bytes) {
    unsigned nsplit = ((unsigned)device_sm_count() + KVH - 1) / KVH;
    const unsigned tiles = (ctx + 31) / 32;
    static_assert(kMaxSplits <= 32, "the merge gives every split a lane");
    if (nsplit > tiles) nsplit = tiles;
    if (nsplit > kMaxSplits) nsplit = kMaxSplits;
    const size_t per_split = (size_t)H * (dh + 2) * sizeof(float);
    const size_t fit = scratch_bytes / per_split;
    if (nsplit > fit) nsplit = (unsigned)fit;
    return nsplit;
}

bool launch_attn_fused(const float* qkv, void* kc, void* vc, bool half_cache, float* scratch, size_t scratch_bytes, float* out,
                       unsigned H, unsigned KVH, unsigned dh, unsigned ctx, float scale, const float* tbl, unsigned tbl_entries,
                       const int* state, cudaStream_t st) {
    if (dh != 64 && dh != 128) return fail("attention: head dim %u unsupported (64 or 128)", dh);
    if (!H || !KVH || H % KVH || KVH > 1024) return fail("attention: bad head counts");
    const unsigned nsplit = attn_fused_splits(H, KVH, dh, ctx, scratch_bytes);
    if (!nsplit) return fail("attention: scratch too small for one split");
    unsigned* counters = attn_counters();
    if (!counters) return fail("attention: counter allocation failed");
    float* part = scratch;
    float* stat = scratch + (size_t)nsplit * H * dh;
    const dim3 grid(KVH, nsplit);
    const unsigned REP = H / KVH;
    bool ok;
    if (half_cache) ok = dh == 128 ? launch_rep<__half, 4>(REP, grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_entries, state)
                                   : launch_rep<__half, 2>(REP, grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_entries, state);
    else ok = dh == 128 ? launch_rep<float, 4>(REP, grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_entries, state)
                        : launch_rep<float, 2>(REP, grid, st, qkv, kc, vc, part, stat, counters, out, H, KVH, ctx, scale, tbl, tbl_entries, state);
    if (!ok) return false;
    note_launch();
    return check_launch("attn_fused");
}

}  // namespace tmc
