// attn_decode.cu — GQA split-K decode attention of one token over a K/V cache.
//
// CUDA form of the reference's attn_decode_gqa(_h) + attn_decode_combine (tensormark/metal.h:2739-2859, host side
// 4153-4222). All arithmetic is fp32.
//
// Bound: HBM, 2 * allow * KVH * dh cache elements read once. A CTA serves the REP query heads that share one K/V head
// over a range of positions, one CTA per SM. The rows of a K/V head are contiguous, so a producer thread streams them
// in 32 KB pieces (bulk copies into a ring of stages, some 190 KB in flight per SM) and nothing but the ring
// limits the bytes in flight: the kernel this replaced read each row with a 2-byte-per-lane load, reduced every score
// with five shuffles and waited for each position in turn (32 / 8 heads of 128, 8191 fp16 positions: 113.8 us, now 14.0 with K and
// V from HBM, whose bytes alone take 5.1, and 11.9 with K and V in L2).
//   * A warp takes 2 KB of K and of V of every stage (4 loads of 16 bytes per lane, the lanes of a row side by side) and
//     keeps its own running maximum and sums: no barrier between warps until the range is finished.
//   * The products of 4 loads x REP heads are summed over a row's lanes by a transposing butterfly (each step halves the
//     values a lane keeps), after which a lane holds the scores it will exponentiate.
//   * fp32 pairs in fma.rn.f32x2 for q k and p v.
// Partials (max, sum, unnormalised output per split) are merged by a second kernel or, where the calls are short, in the same
// launch by the CTAs of a cluster.
#include "common.cuh"
#include "bulk.cuh"
#include "glue.h"
#include "per_device.h"

#include <cstdlib>
#include <cuda_fp16.h>
#include <math_constants.h>
#include <type_traits>

namespace tmc {
namespace {

template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    static const bool on = [] { const char* e = std::getenv("TM_GLUE_PDL"); return !(e && *e == '0'); }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = on ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---- the streaming kernel ------------------------------------------------------------------------------------------
constexpr int kLoads = 4;                                   // 16-byte loads per lane, of K and of V, per stage

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint4 lds16(uint32_t p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p));
    return v;
}
// the 16 bytes of a load as fp32 pairs
template <typename T> struct Elems;
template <> struct Elems<__half> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void pairs(const uint4 v, uint64_t (&o)[4]) {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i])); o[i] = pack2(f.x, f.y); }
    }
};
template <> struct Elems<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void pairs(const uint4 v, uint64_t (&o)[2]) {
        o[0] = pack2(__uint_as_float(v.x), __uint_as_float(v.y)); o[1] = pack2(__uint_as_float(v.z), __uint_as_float(v.w));
    }
};
// More heads want more registers per thread, so fewer warps (with the producer 20, 16 or 8 to the register file's
// eyes: 96, 128 or 255 registers each), fewer bytes per stage and more stages.
template <int REP> struct Split {
    static constexpr int Warps = REP == 8 ? 7 : REP == 4 ? 12 : 16, Stages = REP == 8 ? 7 : REP == 4 ? 4 : 3;
    static constexpr uint32_t Half = Warps * kLoads * 512, Smem = Stages * 2 * Half;      // bytes of K (or V) per stage; of the ring
};

// A wait ran out. status is null in a process that has not initialised the library: there the outputs, which are NaN, have to tell.
__device__ __forceinline__ void note_gone(int* status) {
    if (status) *(volatile int*)status = 1;
}

// The producer leaves when the copies of its last stages have landed, whether or not the warps that they are for still wait: what
// a warp gives up on may come later, and the CTA's shared memory must be its own until then. The first copy that does not come
// within the limit ends the waiting. Out of line, with its flag in shared memory and the count kept outside the loop, it costs nothing
// (8191 fp16 positions of 32 / 8 heads 13.04 us without and with it; a counter in the loop and a flag on the stack: 13.13).
template <uint32_t STAGES>
__device__ __noinline__ void land(uint32_t full, uint32_t issued, int* late) {
#pragma unroll 1
    for (uint32_t i = issued > STAGES ? issued - STAGES : 0u; i < issued; ++i) (void)mbar_wait_slow(full + 8u * (i % STAGES), i / STAGES & 1u, late, kWaitLimitNs);
}

// CLUSTER: the splits of a K/V head are one cluster (1, gridDim.y) whose CTAs merge through distributed shared memory; part is
// then the output itself and stat is not used. Else every split leaves a partial for the merging kernel. In short calls the
// two launches and the way of the partials through L2 are most of the time (32 / 8 heads of 128, 300 fp16 positions: 7.1 us with the
// merging kernel, 6.3 us in one launch); attn_plan.h says where the line lies, some 500 positions for these heads.
template <typename T, int DH, int REP, bool CLUSTER>
__global__ void __launch_bounds__(32 * (Split<REP>::Warps + 1), 1)
attn_stream_kernel(const float* q, const T* kc, const T* vc, float* part, float* stat, uint32_t H, uint32_t ctx, uint32_t allow,
                   uint32_t chunk, float scale, const int* st, int* status) {
    constexpr int NW = Split<REP>::Warps, kStages = Split<REP>::Stages, N = Elems<T>::N, NP = N / 2;         // elements and pairs per lane and load
    constexpr int LR = DH / N, RW = 32 / LR;                                 // lanes per row, rows per load of a warp
    constexpr int PW = kLoads * RW, TP = NW * PW;                            // positions per warp and per stage
    constexpr uint32_t ROW = DH * sizeof(T), HALF = Split<REP>::Half;          // bytes of a row; of K (or V) per stage
    constexpr int NV = kLoads * REP, NVL = NV >= LR ? NV / LR : 1, DUP = NV >= LR ? 1 : LR / NV;   // scores per row group; per lane; lanes that hold the same one
    static_assert(TP * ROW == HALF, "a stage is whole rows");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[2 * kStages];
    __shared__ int gone, late;
    __shared__ __align__(16) float pbuf[NW][PW][REP];                        // a warp's weights of its positions
    __shared__ __align__(16) float cbuf[NW][REP];                            // its correction factors
    __shared__ float sm_m[NW][REP], sm_l[NW][REP];
    __shared__ float2 cta_ml[REP];                                           // CLUSTER: this split's maximum and sum per head
    float* const cta_o = reinterpret_cast<float*>(smem) + NW * REP * DH;     // and its output, behind those of its warps in the ring
    static_assert((NW + 1) * REP * DH * sizeof(float) <= Split<REP>::Smem, "the outputs fit into the ring");
    __shared__ __align__(16) uint4 nothing;                                  // what a lane without a row multiplies its weight 0 by
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        nothing = make_uint4(0u, 0u, 0u, 0u);
        for (int s = 0; s < kStages; ++s) { mbar_init(smem_u32(&bars[s]), 1); mbar_init(smem_u32(&bars[kStages + s]), NW); }
        gone = 0; late = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_enter();
    if (st) {                                               // chain: attend [0, position] with the grid's fixed split count
        allow = min((uint32_t)st[0] + 1u, ctx);
        chunk = (allow + gridDim.y - 1) / gridDim.y;
    }
    const uint32_t kv = blockIdx.x, split = blockIdx.y;
    const uint32_t p0 = min(allow, split * chunk), p1 = min(allow, p0 + chunk), tiles = (p1 - p0 + TP - 1) / TP;
    const uint32_t ring = smem_u32(smem), full = smem_u32(bars), empty = full + 8u * kStages;
    __syncthreads();

    if (warp == NW) {
        if (lane == 0) {
            const uint8_t* kb = reinterpret_cast<const uint8_t*>(kc + ((size_t)kv * ctx + p0) * DH);
            const uint8_t* vb = reinterpret_cast<const uint8_t*>(vc + ((size_t)kv * ctx + p0) * DH);
            uint32_t s = 0, par = 1, issued = tiles;
            for (uint32_t t = 0; t < tiles; ++t) {
                if (!mbar_wait(empty + 8u * s, par, &gone)) { note_gone(status); issued = t; break; }
                const uint32_t bytes = min((uint32_t)TP, p1 - p0 - t * TP) * ROW, bar = full + 8u * s, at = ring + s * 2u * HALF;
                mbar_expect_tx(bar, 2u * bytes);
                bulk_g2s(at, kb + (size_t)t * HALF, bytes, bar);
                bulk_g2s(at + HALF, vb + (size_t)t * HALF, bytes, bar);
                if (++s == (uint32_t)kStages) { s = 0; par ^= 1u; }
            }
            land<(uint32_t)kStages>(full, issued, &late);
        }
    } else {
        const uint32_t gl = (uint32_t)lane % LR, rg = (uint32_t)lane / LR;   // place in a row, row of the load
        uint64_t q2[REP][NP];
#pragma unroll
        for (int r = 0; r < REP; ++r)
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                const float* qr = q + (size_t)(kv * REP + r) * DH + gl * N + 2 * j;
                q2[r][j] = pack2(qr[0] * scale, qr[1] * scale);
            }
        // which scores this lane holds after the butterfly: flattened index load * REP + head = gl / DUP * NVL + k
        const uint32_t first = gl / DUP * NVL;
        float m[NVL], l[NVL];
        uint64_t acc[REP][NP];
#pragma unroll
        for (int k = 0; k < NVL; ++k) { m[k] = -CUDART_INF_F; l[k] = 0.f; }
#pragma unroll
        for (int r = 0; r < REP; ++r)
#pragma unroll
            for (int j = 0; j < NP; ++j) acc[r][j] = 0ull;
        uint32_t s = 0, par = 0;
        bool ok = true;
        for (uint32_t t = 0; t < tiles; ++t) {
            const uint32_t np = min((uint32_t)TP, p1 - p0 - t * TP);         // positions of this stage
            if (!mbar_wait(full + 8u * s, par, &gone)) ok = false;
            const uint32_t at = ring + s * 2u * HALF;
            uint32_t off[kLoads];                                            // rows past the end: the last row's K again, whose score is dropped
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                const uint32_t pos = (uint32_t)(warp * kLoads + i) * RW + rg;
                off[i] = min(pos, np - 1u) * ROW + gl * 16u;
            }
            float v[NV];
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                uint64_t k2[NP];
                Elems<T>::pairs(lds16(at + off[i]), k2);
#pragma unroll
                for (int r = 0; r < REP; ++r) {
                    uint64_t a = mul2(q2[r][0], k2[0]);
#pragma unroll
                    for (int j = 1; j < NP; ++j) a = fma2(q2[r][j], k2[j], a);
                    const float2 f = unpack2(a);
                    v[i * REP + r] = f.x + f.y;
                }
            }
            // transposing butterfly over the LR lanes of a row
            {
                int n = NV;
#pragma unroll
                for (int o = LR / 2; o; o >>= 1) {
                    if (n > 1) {
                        n >>= 1;
                        const bool up = gl & (uint32_t)o;
#pragma unroll
                        for (int k = 0; k < NV / 2; ++k)
                            if (k < n) {
                                const float keep = up ? v[k + n] : v[k], give = up ? v[k] : v[k + n];
                                v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                            }
                    } else {
                        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
                    }
                }
            }
            // softmax of this warp's positions, per head
            float mn[NVL];
            bool moved = false;
#pragma unroll
            for (int k = 0; k < NVL; ++k) {
                const uint32_t idx = first + k, pos = (uint32_t)(warp * kLoads) * RW + idx / REP * RW + rg;
                if (pos >= np) v[k] = -CUDART_INF_F;
                float x = v[k];
                constexpr uint32_t rbits = NV >= LR ? (uint32_t)(REP > NVL ? REP / NVL - 1 : 0) : (uint32_t)((REP - 1) * DUP);   // lane bits that name the head
#pragma unroll
                for (int o = 16; o; o >>= 1)
                    if (!((uint32_t)o & rbits)) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
                mn[k] = x;
            }
            if constexpr (NVL > REP) {                                       // several of a lane's scores are of one head
#pragma unroll
                for (int k = 0; k < NVL; ++k)
#pragma unroll
                    for (int h = k % REP; h < NVL; h += REP) mn[k] = fmaxf(mn[k], mn[h]);
            }
            float corr[NVL];
#pragma unroll
            for (int k = 0; k < NVL; ++k) {
                mn[k] = fmaxf(mn[k], m[k]);
                moved = moved || mn[k] > m[k];
                corr[k] = m[k] == -CUDART_INF_F ? 0.f : __expf(m[k] - mn[k]);
                v[k] = v[k] == -CUDART_INF_F ? 0.f : __expf(v[k] - mn[k]);
                l[k] = l[k] * corr[k] + v[k];
                m[k] = mn[k];
            }
            __syncwarp();                                                    // the last stage's weights have been read
#pragma unroll
            for (int k = 0; k < NVL; ++k) {
                const uint32_t idx = first + k;
                if (gl % DUP == 0) pbuf[warp][idx / REP * RW + rg][idx % REP] = v[k];
                if (gl % DUP == 0 && idx < REP && rg == 0) cbuf[warp][idx] = corr[k];
            }
            __syncwarp();
            if (__any_sync(0xffffffffu, moved)) {                            // rare after the first stages
#pragma unroll
                for (int r = 0; r < REP; ++r) {
                    const float c = cbuf[warp][r];
#pragma unroll
                    for (int j = 0; j < NP; ++j) acc[r][j] = mul2(acc[r][j], pack2(c, c));
                }
            }
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                uint64_t v2[NP];                                             // past the end zeros: the last row's V may be infinite
                Elems<T>::pairs(lds16((uint32_t)(warp * kLoads + i) * RW + rg < np ? at + HALF + off[i] : smem_u32(&nothing)), v2);
                float pw[REP];
                if constexpr (REP % 4 == 0) {
#pragma unroll
                    for (int r = 0; r < REP; r += 4) *reinterpret_cast<float4*>(&pw[r]) = *reinterpret_cast<const float4*>(&pbuf[warp][i * RW + rg][r]);
                } else {
#pragma unroll
                    for (int r = 0; r < REP; ++r) pw[r] = pbuf[warp][i * RW + rg][r];
                }
#pragma unroll
                for (int r = 0; r < REP; ++r) {
                    const uint64_t w = pack2(pw[r], pw[r]);
#pragma unroll
                    for (int j = 0; j < NP; ++j) acc[r][j] = fma2(w, v2[j], acc[r][j]);
                }
            }
            __syncwarp();
            mbar_arrive_if(empty + 8u * s, lane == 0);
            if (++s == (uint32_t)kStages) { s = 0; par ^= 1u; }
        }
        // a head's sum lies over the lanes that do not name it and are not duplicates
        if constexpr (NVL > REP) {
#pragma unroll
            for (int k = REP; k < NVL; ++k) l[k % REP] += l[k];
        }
#pragma unroll
        for (int k = 0; k < (NVL < REP ? NVL : REP); ++k) {
            constexpr uint32_t rbits = NV >= LR ? (uint32_t)(REP > NVL ? REP / NVL - 1 : 0) : (uint32_t)((REP - 1) * DUP);
            float x = l[k];
#pragma unroll
            for (int o = 16; o; o >>= 1)
                if (!((uint32_t)o & rbits) && o >= DUP) x += __shfl_xor_sync(0xffffffffu, x, o);
            const uint32_t idx = first + k;
            if (gl % DUP == 0 && idx < REP && rg == 0) { sm_m[warp][idx] = m[k]; sm_l[warp][idx] = x; }
        }
#pragma unroll
        for (int r = 0; r < REP; ++r)
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                float2 f = unpack2(acc[r][j]);
#pragma unroll
                for (int o = LR; o < 32; o <<= 1) { f.x += __shfl_xor_sync(0xffffffffu, f.x, o); f.y += __shfl_xor_sync(0xffffffffu, f.y, o); }
                acc[r][j] = pack2(f.x, f.y);
            }
        __syncwarp();
        if (!ok) {                                                           // rows that never came were multiplied: no number may pass for the result
            note_gone(status);
            for (int r = 0; r < REP; ++r) sm_l[warp][r] = CUDART_NAN_F;
        }
        // the ring is free once every warp is through with it: the warps' outputs go there
        asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
        float* out = reinterpret_cast<float*>(smem);                         // [NW][REP][DH]
        if (rg == 0) {
#pragma unroll
            for (int r = 0; r < REP; ++r)
#pragma unroll
                for (int j = 0; j < NP; ++j) *reinterpret_cast<float2*>(out + ((size_t)warp * REP + r) * DH + gl * N + 2 * j) = unpack2(acc[r][j]);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
        for (uint32_t i = threadIdx.x; i < (uint32_t)(REP * DH); i += NW * 32) {
            const uint32_t r = i / DH, d = i % DH, head = kv * REP + r;
            float M = -CUDART_INF_F;
#pragma unroll
            for (int w = 0; w < NW; ++w) M = fmaxf(M, sm_m[w][r]);
            float o = 0.f, L = 0.f;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const float f = sm_m[w][r] == -CUDART_INF_F ? 0.f : __expf(sm_m[w][r] - M);
                o = fmaf(f, out[((size_t)w * REP + r) * DH + d], o);
                L = fmaf(f, sm_l[w][r], L);
            }
            if constexpr (CLUSTER) {
                cta_o[i] = o;
                if (d == 0) cta_ml[r] = make_float2(M, L);
            } else {
                part[((size_t)split * H + head) * DH + d] = o;
                if (d == 0) { stat[((size_t)split * H + head) * 2] = M; stat[((size_t)split * H + head) * 2 + 1] = L; }
            }
        }
    }
    if constexpr (CLUSTER) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const uint32_t nsplit = gridDim.y, per = (uint32_t)(REP * DH) / nsplit;       // every CTA merges its share of the outputs: both are powers of two
        for (uint32_t i = split * per + threadIdx.x; i < (split + 1u) * per; i += blockDim.x) {
            const uint32_t at_o = smem_u32(cta_o) + 4u * i, at_ml = smem_u32(cta_ml) + 8u * (i / DH);
            float2 ml[kMaxCluster];
            float x[kMaxCluster], M = -CUDART_INF_F, o = 0.f, L = 0.f;
#pragma unroll
            for (uint32_t k = 0; k < kMaxCluster; ++k)
                if (k < nsplit) {
                    uint32_t a, b;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(at_ml), "r"(k));
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(at_o), "r"(k));
                    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(ml[k].x), "=f"(ml[k].y) : "r"(a) : "memory");
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[k]) : "r"(b) : "memory");
                }
#pragma unroll
            for (uint32_t k = 0; k < kMaxCluster; ++k)
                if (k < nsplit) M = fmaxf(M, ml[k].x);
#pragma unroll
            for (uint32_t k = 0; k < kMaxCluster; ++k)
                if (k < nsplit) {
                    const float f = ml[k].x == -CUDART_INF_F ? 0.f : __expf(ml[k].x - M);
                    o = fmaf(f, x[k], o);
                    L = fmaf(f, ml[k].y, L);
                }
            part[(size_t)kv * (REP * DH) + i] = o * (1.0f / L);
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // nobody leaves while its shared memory is read
    }
}

// ---- caches off the 16-byte grid ---------------------------------------------------------------------------------------
// grid (KVH, nsplit), 4 warps. A CTA serves the REP query heads that share one KV
// head over positions [split*chunk, min(allow, (split+1)*chunk)). Each warp walks
// its positions with an online softmax; a lane owns dh/32 consecutive dims, so one
// K or V row is a single coalesced read. The four warps' states are merged in
// shared memory and the CTA writes one unnormalised partial per query head:
// part[(split*H + head)*dh + d] and stat[(split*H + head)*2] = (max, sum).
template <typename T, int DPL, int REP>
__global__ void __launch_bounds__(128) attn_split_kernel(const float* q, const T* kc,
                                                          const T* vc, float* part,
                                                          float* stat, uint32_t H, uint32_t ctx,
                                                          uint32_t allow, uint32_t chunk, float scale,
                                                          const int* st) {
    pdl_enter();
    constexpr int dh = DPL * 32;
    if (st) {                                               // chain: attend [0, position] with the grid's fixed split count
        allow = min((uint32_t)st[0] + 1u, ctx);
        chunk = (allow + gridDim.y - 1) / gridDim.y;
    }
    const uint32_t kv = blockIdx.x, split = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t p0 = split * chunk, p1 = min(allow, p0 + chunk);
    __shared__ float sm_acc[4][REP][dh];
    __shared__ float sm_m[4][REP], sm_l[4][REP];

    float qr[REP][DPL];
#pragma unroll
    for (int r = 0; r < REP; ++r)
#pragma unroll
        for (int d = 0; d < DPL; ++d) qr[r][d] = q[(size_t)(kv * REP + r) * dh + lane * DPL + d] * scale;

    float m[REP], l[REP], acc[REP][DPL];
#pragma unroll
    for (int r = 0; r < REP; ++r) {
        m[r] = -CUDART_INF_F; l[r] = 0.f;
#pragma unroll
        for (int d = 0; d < DPL; ++d) acc[r][d] = 0.f;
    }
    const T* kbase = kc + (size_t)kv * ctx * dh + lane * DPL;
    const T* vbase = vc + (size_t)kv * ctx * dh + lane * DPL;
    for (uint32_t p = p0 + warp; p < p1; p += 4) {
        float kf[DPL], vf[DPL];
#pragma unroll
        for (int d = 0; d < DPL; ++d) { kf[d] = (float)kbase[(size_t)p * dh + d]; vf[d] = (float)vbase[(size_t)p * dh + d]; }
#pragma unroll
        for (int r = 0; r < REP; ++r) {
            float s = 0.f;
#pragma unroll
            for (int d = 0; d < DPL; ++d) s = fmaf(qr[r][d], kf[d], s);
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const float mn = fmaxf(m[r], s);
            const float corr = __expf(m[r] - mn), pw = __expf(s - mn);
            l[r] = l[r] * corr + pw;
#pragma unroll
            for (int d = 0; d < DPL; ++d) acc[r][d] = fmaf(acc[r][d], corr, pw * vf[d]);
            m[r] = mn;
        }
    }
#pragma unroll
    for (int r = 0; r < REP; ++r) {
        if (lane == 0) { sm_m[warp][r] = m[r]; sm_l[warp][r] = l[r]; }
#pragma unroll
        for (int d = 0; d < DPL; ++d) sm_acc[warp][r][lane * DPL + d] = acc[r][d];
    }
    __syncthreads();
    // merge the four warps: thread t handles dims t, t+128, ... of every head
    for (int r = 0; r < REP; ++r) {
        float M = -CUDART_INF_F;
#pragma unroll
        for (int w = 0; w < 4; ++w) M = fmaxf(M, sm_m[w][r]);
        float Lsum = 0.f;
        float f[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) { f[w] = sm_m[w][r] == -CUDART_INF_F ? 0.f : __expf(sm_m[w][r] - M); Lsum += f[w] * sm_l[w][r]; }
        const uint32_t head = kv * REP + r;
        for (int d = threadIdx.x; d < dh; d += 128) {
            float o = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) o += f[w] * sm_acc[w][r][d];
            part[((size_t)split * H + head) * dh + d] = o;
        }
        if (threadIdx.x == 0) { stat[((size_t)split * H + head) * 2] = M; stat[((size_t)split * H + head) * 2 + 1] = Lsum; }
    }
}


// out[head][d] = sum_s e^(m_s - M) part_s[d] / sum_s e^(m_s - M) l_s. One CTA per head; bound by its chain of round trips to
// L2. Four threads per dim take every fourth split, so 40 partials are on their way at a time, while a lane per split reads
// its maximum and sum at once and works out the weights. A thread per dim, 20 partials at a time and the maxima read
// before the sums, against this, us with the split kernel, 8191 fp16 positions, K and V in L2 (from HBM): 32 / 8 heads of 128 (18 splits)
// 13.5 / 11.9 (15.5 / 14.0); 32 / 4 of 64 (37) 11.0 / 9.4 (12.0 / 10.6); 8 / 1 of 128 (147) 22.4 / 11.7 (22.9 / 12.1); 40 / 40 of 128 (3)
// 31.0 / 31.0 (31.1 / 31.0).
constexpr uint32_t kMergeGroups = 4;
__global__ void __launch_bounds__(kMergeGroups * 128) attn_combine_kernel(const float* part, const float* stat, float* out, uint32_t H, uint32_t dh, uint32_t nsplit) {
    constexpr uint32_t BATCH = 10, G = kMergeGroups, MOST = 256;
    __shared__ float sums[G - 1][128];
    __shared__ float wsum[MOST];
    __shared__ float inv;
    pdl_enter();
    const uint32_t head = blockIdx.x, lane = threadIdx.x & 31u, d = threadIdx.x % dh, grp = threadIdx.x / dh;      // G * dh threads
    float v[BATCH];
    auto request = [&](uint32_t s0) {
#pragma unroll
        for (uint32_t k = 0; k < BATCH; ++k)
            if (s0 + G * k + grp < nsplit) v[k] = __ldcg(part + ((size_t)(s0 + G * k + grp) * H + head) * dh + d);
    };
    request(0);
    if (threadIdx.x < 32) {
        float2 ml[MOST / 32];
        float M = -CUDART_INF_F, L = 0.f;
#pragma unroll
        for (uint32_t i = 0; i < MOST / 32; ++i) {
            const uint32_t s = lane + 32u * i;
            const float* at = stat + ((size_t)s * H + head) * 2;             // scratch is on 4 bytes
            ml[i] = s < nsplit ? make_float2(__ldcg(at), __ldcg(at + 1)) : make_float2(-CUDART_INF_F, 0.f);
        }
#pragma unroll
        for (uint32_t i = 0; i < MOST / 32; ++i) M = fmaxf(M, ml[i].x);
#pragma unroll
        for (int o = 16; o; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
        for (uint32_t i = 0; i < MOST / 32; ++i) {
            const uint32_t s = lane + 32u * i;
            if (s >= nsplit) continue;
            const float w = ml[i].x == -CUDART_INF_F ? 0.f : __expf(ml[i].x - M);
            wsum[s] = w;
            L = fmaf(w, ml[i].y, L);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        if (lane == 0) inv = 1.0f / L;
    }
    __syncthreads();
    float o = 0.f;
    for (uint32_t s0 = 0; s0 < nsplit; s0 += G * BATCH) {
        if (s0) request(s0);
#pragma unroll
        for (uint32_t k = 0; k < BATCH; ++k)
            if (s0 + G * k + grp < nsplit) o = fmaf(wsum[s0 + G * k + grp], v[k], o);
    }
    if (grp) sums[grp - 1][d] = o;
    __syncthreads();
    if (grp) return;
#pragma unroll
    for (uint32_t i = 0; i < G - 1; ++i) o += sums[i][d];
    out[(size_t)head * dh + d] = o * inv;
}

// Function attributes are a device's own: what the launches below prepare, they prepare for the device that is current.
int current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    return dev;
}

template <typename T, int DH, int REP>
bool launch_stream(dim3 grid, cudaStream_t st, const float* q, const T* kc, const T* vc, float* part, float* stat, unsigned H, unsigned ctx,
                   unsigned allow, unsigned chunk, float scale, const int* state) {
    auto* kernel = attn_stream_kernel<T, DH, REP, false>;
    static PerDevice<bool> ready;
    const int dev = current_device();
    if (dev < 0 || dev >= kMaxDevices) return fail("attention: no current CUDA device");
    if (!ready.get(dev, [=](bool&) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Split<REP>::Smem);
            return e == cudaSuccess || fail("attention: shared memory attribute: %s", cudaGetErrorString(e));
        })) return false;
    launch_pdl(kernel, grid, dim3(32 * (Split<REP>::Warps + 1)), Split<REP>::Smem, st, q, kc, vc, part, stat, H, ctx, allow, chunk, scale, state, device_status_word());
    return true;
}

// One launch with a cluster of `cs` splits per K/V head; false (and no error) where the device cannot hold KVH of them at a time.
template <typename T, int DH, int REP>
bool launch_cluster(unsigned cs, unsigned KVH, cudaStream_t st, const float* q, const T* kc, const T* vc, float* out, unsigned H, unsigned ctx,
                    unsigned allow, float scale, const int* state) {
    auto* kernel = attn_stream_kernel<T, DH, REP, true>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(KVH, cs); cfg.blockDim = dim3(32 * (Split<REP>::Warps + 1)); cfg.dynamicSmemBytes = Split<REP>::Smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = cs; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    struct Fits { int clusters[5]; };                       // of 1, 2, 4, 8, 16 CTAs, that run at a time
    static PerDevice<Fits> device;
    const Fits* fits = device.get(current_device(), [&](Fits& f) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Split<REP>::Smem) != cudaSuccess ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { cudaGetLastError(); return false; }
        cudaLaunchConfig_t c = cfg;
        cudaLaunchAttribute a = at[0];
        c.attrs = &a; c.numAttrs = 1;
        for (int i = 0; i < 5; ++i) {
            a.val.clusterDim.y = 1u << i;
            c.gridDim = dim3(1, 1u << i);
            if (cudaOccupancyMaxActiveClusters(&f.clusters[i], kernel, &c) != cudaSuccess) { cudaGetLastError(); f.clusters[i] = 0; }
        }
        return true;
    });
    int i = 0;
    while (1u << i < cs) ++i;
    if (!fits || fits->clusters[i] < (int)KVH) return false;
    static const bool pdl = [] { const char* e = std::getenv("TM_GLUE_PDL"); return !(e && *e == '0'); }();
    cfg.numAttrs = pdl ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, q, kc, vc, out, (float*)nullptr, (uint32_t)H, (uint32_t)ctx, (uint32_t)allow, (uint32_t)attn_cdiv(allow, cs), scale, state, device_status_word());
    return true;
}
// One K/V head per grid column. The streaming kernel copies whole rows in bulk and wants the caches on 16-byte boundaries;
// caches on any other address take the element-wise one.
template <typename T, int DH>
bool launch_splits(unsigned sms, unsigned REP, unsigned KVH, AttnSplits sp, cudaStream_t st, const float* q, const T* kc, const T* vc, float* part, float* stat, float* out,
                   unsigned H, unsigned ctx, unsigned allow, float scale, const int* state, bool* merged) {
    static const bool one = [] { const char* e = std::getenv("TM_ATTN_CLUSTER"); return !(e && *e == '0'); }();   // A/B knob
    const dim3 grid(KVH, sp.nsplit);
    const bool bulk = (uintptr_t)kc % 16 == 0 && (uintptr_t)vc % 16 == 0;
    bool ok = true;
    *merged = false;
    auto go = [&](auto rep) {
        constexpr int R = decltype(rep)::value;
        if (bulk && one) {
            const AttnClusters c = attn_clusters(sms, KVH, R, DH, sizeof(T), allow, grid.y);
            for (unsigned cs = c.cs; cs && attn_cdiv(allow, cs) <= c.longest && !*merged; cs >>= 1)
                *merged = launch_cluster<T, DH, R>(cs, KVH, st, q, kc, vc, out, H, ctx, allow, scale, state);
            if (*merged) return;
        }
        if (bulk) ok = launch_stream<T, DH, R>(grid, st, q, kc, vc, part, stat, H, ctx, allow, sp.chunk, scale, state);
        else launch_pdl(attn_split_kernel<T, DH / 32, R>, grid, dim3(128), 0, st, q, kc, vc, part, stat, H, ctx, allow, sp.chunk, scale, state);
    };
    switch (REP) {
        case 1: go(std::integral_constant<int, 1>{}); break;
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 4: go(std::integral_constant<int, 4>{}); break;
        case 8: go(std::integral_constant<int, 8>{}); break;
        default: return fail("attention: REP=%u unsupported (1, 2, 4 or 8)", REP);
    }
    if (!ok) return false;
    note_launch();
    return check_launch("attn_split");
}

}  // namespace

AttnPlan plan_attention(unsigned H, unsigned KVH, unsigned dh, unsigned allow, size_t scratch_bytes) {
    return plan_attention_sms((unsigned)device_sm_count(), H, KVH, dh, allow, scratch_bytes);
}

bool launch_attention(const float* q, const void* kc, const void* vc, bool half_cache, float* scratch, float* out,
                      unsigned H, unsigned KVH, unsigned dh, unsigned ctx, unsigned allow, float scale, unsigned REP,
                      const AttnPlan& pl, cudaStream_t st, const int* state) {
    if (dh != 64 && dh != 128) return fail("attention: head dim %u unsupported (64 or 128)", dh);
    const AttnSplits sp = attn_splits(pl, KVH, allow, state != nullptr);
    float* part = scratch;
    float* stat = scratch + pl.part_floats;
    bool ok, merged;
    if (half_cache) {
        const __half *k = (const __half*)kc, *v = (const __half*)vc;
        ok = dh == 128 ? launch_splits<__half, 128>(pl.sms, REP, KVH, sp, st, q, k, v, part, stat, out, H, ctx, allow, scale, state, &merged)
                       : launch_splits<__half, 64>(pl.sms, REP, KVH, sp, st, q, k, v, part, stat, out, H, ctx, allow, scale, state, &merged);
    } else {
        const float *k = (const float*)kc, *v = (const float*)vc;
        ok = dh == 128 ? launch_splits<float, 128>(pl.sms, REP, KVH, sp, st, q, k, v, part, stat, out, H, ctx, allow, scale, state, &merged)
                       : launch_splits<float, 64>(pl.sms, REP, KVH, sp, st, q, k, v, part, stat, out, H, ctx, allow, scale, state, &merged);
    }
    if (!ok || merged) return ok;
    launch_pdl(attn_combine_kernel, dim3(H), dim3(kMergeGroups * dh), 0, st, part, stat, out, H, dh, sp.nsplit);
    note_launch();
    return check_launch("attn_combine");
}

}  // namespace tmc
