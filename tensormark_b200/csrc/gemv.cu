// gemv.cu — streaming block-quantized GEMV for sm_100a:  y[N] = W[N x K] * x[K].
//
// Replaces the cooperative-row Metal GEMVs (tensormark/metal.h:359-440 Q4_0,
// 641-679 Q4_1, 708-754 Q5_K, 775-822 Q6_K, and their segmented forms 511-567,
// 915-1078) and adds the Q8_0 kernel the reference GPU lane lacks.
//
// Bound: HBM; every weight byte is read exactly once, at its serialized width. One CTA per SM takes a contiguous range
// of rows. Two to four producer warps stream it through a ring in shared memory with bulk asynchronous copies (cp.async.bulk
// global -> shared, completion on an mbarrier), so the bytes in flight are set by the ring and no thread ever holds a
// weight load in a register; sixteen consumer warps multiply on the integer tensor cores (gemv_tile.cuh has the
// geometry, gemv_lanes.cuh the arithmetic).
//   * x is staged once per CTA into shared memory as block floating point in the MMA's operand layout; the weight
//     stream is already running then: producers do not wait for the preceding kernel (programmatic dependent launch).
//   * A row's sums meet in a fixed order that depends on K and the format only, so a row's result does not depend on
//     the grid or on whether it was reached through a segment table: the segmented launch is bit-identical to separate
//     launches (the property tensormark/metal.h:504-510 requires).
//   * Rows that start on any even address are served: a row's copy starts at the 16-byte boundary below it and the
//     lanes read from the remainder on (AL = false). Such rows used to be multiplied by x in fp32; here x keeps four
//     planes for them, which holds an fp32 x to its last bits. Odd addresses, TQ2 and an x of more than kMaxPlaneK take
//     gemv_generic, a plain byte-granular kernel with the same per-row arithmetic contract (tolerance-level, not bitwise, agreement).
#include "common.cuh"
#include "gemv_tile.cuh"
#include "share_count.h"

#include <cstdlib>

namespace tmc {

namespace {

struct GemvParams {
    const uint8_t* W;
    const float* x;
    float* y;
    uint32_t N, K, row_bytes;
    uint32_t slots, rows_per_cta;
    TileGeom ge;
    // optional fusions (decode chain): a transform of x while it is staged, and y += instead of y =
    const float* x2;            // x_op 1: rmsnorm weights; x_op 2: the "up" vector
    float eps;
    uint32_t x_op;              // 0 plain, 1 x*rsqrt(mean(x^2)+eps)*x2, 2 silu(x)*x2
    uint32_t accumulate;
    SegTable seg;
    Exchange xc;                // row-sharded models: wait for peers before x, push y to peers after
    unsigned long long* trace;  // kernel timeline, nullptr when off
    int* status;
    // x already in the lanes' form (written once per launch by xprep_kernel): the CTA bulk-copies the image
    // instead of staging x itself. Layout: 16 header words ([0] = the RMSNorm
    // factor as a float, 1.0 when none), then the groups.
    const uint32_t* xq;
    uint32_t* share;            // the same image, made by this launch's CTAs together (GemvFuse::share)
    unsigned* share_ctr;
    uint32_t share_want;        // the counter's value when it is complete
    unsigned long long x_ns;            // how long x may take once the preceding kernel is through, and a row after that
    unsigned long long share_ns;        // how long a CTA waits for the others' parts
};

__device__ __forceinline__ const uint8_t* row_ptr(const GemvParams& p, uint32_t row) {
    uint32_t s = 0, start = 0;
    while (s + 1 < p.seg.nseg && row >= p.seg.row_end[s]) { start = p.seg.row_end[s]; ++s; }
    return p.W + p.seg.woff[s] + (size_t)(row - start) * p.row_bytes;
}

// Element of y that receives `row` (segments may land at separate offsets of y).
__device__ __forceinline__ uint32_t y_index(const GemvParams& p, uint32_t row) {
    uint32_t s = 0, start = 0;
    while (s + 1 < p.seg.nseg && row >= p.seg.row_end[s]) { start = p.seg.row_end[s]; ++s; }
    return p.seg.yoff[s] + (row - start);
}

// One CTA stages the whole vector x (K activations) for a consumer of format CDT into `out` (global memory: 16 header
// words, then the units), and writes the RMSNorm factor into out[0]. Warp w takes groups w, w + nwarps, ... so the
// sum of squares is added in the same order as when a GEMV CTA stages x for itself.
template <int CDT>
__device__ __forceinline__ void stage_vector(uint32_t* out, const float* x, const float* x2, uint32_t x_op, float eps, uint32_t K, float* red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const uint32_t ngroups = (K + 255u) / 256u;
    float ss = stage_groups<CDT>(out + kXqHeaderWords, nullptr, x, x2, x_op, K, (uint32_t)warp, ngroups, (uint32_t)nwarps, lane);
    if (x_op == 1u) {
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) red[warp] = ss;
        __syncthreads();
        if (threadIdx.x == 0) {
            float tot = 0.f;
            for (int w = 0; w < nwarps; ++w) tot += red[w];
            out[0] = __float_as_uint(1.0f / sqrtf(tot / (float)K + eps));
        }
    } else if (threadIdx.x == 0) {
        out[0] = __float_as_uint(1.0f);
    }
}
// x in unit form, once per launch. RMSNorm needs the
// sum over the whole vector and runs as ONE CTA of 16 warps; the other transforms have no cross-group term and run
// as many small CTAs as there are groups to cover.
template <int CDT>
__global__ void __launch_bounds__(512) xprep_kernel(uint32_t* out, const float* x, const float* x2, uint32_t x_op, float eps, uint32_t K,
                                                    const Exchange xc, int* status) {
    __shared__ float red[16];
    // The GEMV that follows may become resident and prefetch its weights at once; it waits for this grid itself.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (x_op == 1u)                                        // norm weights: static, and out of L2 since the last token
        for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 32u; i < K; i += gridDim.x * blockDim.x * 32u)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(x2 + i) : "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    exchange_wait(xc, status);
    if (gridDim.x == 1) { stage_vector<CDT>(out, x, x2, x_op, eps, K, red); return; }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const uint32_t ngroups = (K + 255u) / 256u, g = blockIdx.x * nwarps + warp;
    if (g < ngroups) (void)stage_groups<CDT>(out + kXqHeaderWords, nullptr, x, x2, x_op, K, g, g + 1, 1u, lane);
    if (blockIdx.x == 0 && threadIdx.x == 0) out[0] = __float_as_uint(1.0f);
}


// Shared memory: [x image and a group of zeros][the ring's barriers][ring].
__host__ __device__ inline uint32_t x_smem(const TileGeom& g, bool aligned) { return x_image_bytes(g.ngroups) * (aligned ? 1u : 2u); }
static_assert(kRingBarBytes % 128 == 0, "the ring starts on a 128-byte boundary");

template <int DT, bool AL>
__global__ void __launch_bounds__(gemv_threads(DT), 1) gemv_stream(const GemvParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float red[kConsumers];
    __shared__ Patience patience;
    __shared__ __align__(8) uint64_t xbar;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long* tr = nullptr;                       // this launch's timeline record (CTA 0, thread 0 only)
    if (p.trace && blockIdx.x == 0 && threadIdx.x == 0) {
        const unsigned long long slot = atomicAdd(p.trace, 1ull);
        if (slot < (unsigned long long)kTraceLaunches) {
            tr = p.trace + 1 + slot * kTraceWords;
            tr[0] = global_ns();
            tr[4] = ((unsigned long long)p.N << 32) | p.K;
            tr[5] = (unsigned long long)DT | ((unsigned long long)p.x_op << 8) | ((unsigned long long)kConsumers << 16) | ((unsigned long long)kTileRows << 24);
        }
    }
    const TileGeom ge = p.ge;
    uint32_t* img = reinterpret_cast<uint32_t*>(smem);
    Ring rg;
    rg.bars = smem_base(smem) + x_smem(ge, AL);
    rg.at = rg.bars + kRingBarBytes;
    rg.slots = p.slots; rg.slot_bytes = ge.slot_bytes; rg.patience = &patience;
    const uint32_t cta_lo = min(p.N, blockIdx.x * p.rows_per_cta), rows = min(p.N, cta_lo + p.rows_per_cta) - cta_lo;

    if (threadIdx.x == 0) {
        rg.init(reducers(DT));
        mbar_init(smem_u32(&xbar), 1);
        patience = {0, p.status, p.x_ns};
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp >= kConsumers + kProducers) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // y (+=) may be what the preceding kernel wrote
        float norm_inv = 1.f;
        float* const y = p.y;
        const uint32_t e0 = p.seg.yoff[0] + cta_lo, x_op = p.x_op, npush = p.xc.npush;
        const bool plain = p.seg.nseg == 1u, add = p.accumulate != 0u;
        RingPos pos{0, 0};
        reduce<reducers(DT)>(rg, pos, ge, rows, (uint32_t)(warp - kConsumers - kProducers), lane,
               [&] {                                         // the sums of squares are in place since before the first item
                   if (p.xq) {
                       norm_inv = red[0];                    // written with the image by whoever staged it
                   } else if (p.x_op == 1u) {
                       float tot = 0.f;                      // fixed order
#pragma unroll
                       for (int w = 0; w < kConsumers; ++w) tot += red[w];
                       norm_inv = 1.0f / sqrtf(tot / (float)p.K + p.eps);
                   }
               },
               [&](uint32_t row, float v) {
                   const uint32_t e = plain ? e0 + row : y_index(p, cta_lo + row);
                   if (x_op == 1u) v *= norm_inv;
                   if (add) v += __ldcg(y + e);              // residual add folded into the store
                   y[e] = v;
                   for (uint32_t q = 0; q < npush; ++q) p.xc.peer_y[q][e] = v;      // a sharded model's peers
               });
    } else if (warp >= kConsumers) {
        // The producers touch only weights and run ahead of everything the consumers wait for.
        RingPos pos{0, 1};
        const bool plain = p.seg.nseg == 1u;
        const uint32_t row_bytes = p.row_bytes;
        const uint8_t* const first = p.W + p.seg.woff[0] + (size_t)cta_lo * row_bytes;
        if (!produce<AL>(rg, pos, ge, rows, row_bytes, (uint32_t)(warp - kConsumers), lane,
                         [&](uint32_t row) { return plain ? first + (size_t)row * row_bytes : row_ptr(p, cta_lo + row); }) && lane == 0) drain(rg);
    } else {
        // RMSNorm weights are read once per token, 4 GB of streamed blocks apart: by then they have left L2, and their
        // DRAM latency would sit between the dependency wait and the first row. They do not depend on the preceding
        // kernel: ask for them now. x itself may still be written by the preceding kernel, but L2 is where its writes
        // land: asking for the lines now costs nothing when they are there and saves the DRAM round trip when not.
        if (!p.xq && !p.share) {
            for (uint32_t i = threadIdx.x * 32u; i < p.K; i += kConsumers * 1024u) {
                if (p.x_op == 1u) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.x2 + i) : "memory");
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p.x + i) : "memory");
            }
        }
        for (uint32_t i = threadIdx.x; i < (uint32_t)kXGroupWords; i += kConsumers * 32) img[ge.ngroups * kXGroupWords + i] = 0u;
        // Everything above touches only weights. x may be written by the preceding kernel in the stream: wait for it
        // here, and let the next kernel start its own weight stream.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        if (p.xc.nwait) {                                    // sharded models: x is complete once every peer has pushed
            if (threadIdx.x == 0) (void)exchange_wait_thread(p.xc, p.status);
            consumer_sync();
        }
        if (tr) tr[1] = global_ns();

        // x image into shared memory: one bulk copy when it was written once for the whole launch, else staged here
        if (p.xq) {
            if (threadIdx.x == 0) {
                const uint32_t xbytes = ge.ngroups * (uint32_t)kXGroupWords * 4u, xb = smem_u32(&xbar);
                mbar_expect_tx(xb, xbytes);
                bulk_g2s(smem_u32(img), p.xq + kXqHeaderWords, xbytes, xb);
                red[0] = __uint_as_float(__ldcg(p.xq));
                if (!mbar_wait(xb, 0, &patience.gone)) *(volatile int*)p.status = 1;
            }
        } else if (AL && p.share) {
            // A part per CTA, read once. The lowest CTAs have them and wait for nobody before they make theirs; the image is
            // complete a few microseconds after the last of those has started. When that is depends on what else the GPU
            // runs (another stream's kernel may hold its SM), so a CTA whose patience (share_ns) ends stages all of x for
            // itself: 4 K more bytes over PCIe, the same bits. (A staging launch ahead of the GEMV cost a second launch and
            // its hand-over: a host call of 256 x 2048 20.7 us, now 19.6.)
            (void)stage_groups<DT>(p.share + kXqHeaderWords, nullptr, p.x, nullptr, 0u, p.K, blockIdx.x + (uint32_t)warp * gridDim.x, ge.ngroups,
                                   (uint32_t)kConsumers * gridDim.x, lane);
            consumer_sync();
            if (threadIdx.x == 0) {
                if (blockIdx.x < ge.ngroups) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.share_ctr) : "memory");
                red[0] = p.share_ns && wait_counter(p.share_ctr, p.share_want, p.share_ns, nullptr) ? 1.f : 0.f;
            }
            consumer_sync();
            if (red[0] != 0.f) {
                const uint4* from = reinterpret_cast<const uint4*>(p.share + kXqHeaderWords);
                for (uint32_t i = threadIdx.x; i < ge.ngroups * (uint32_t)kXGroupWords / 4u; i += kConsumers * 32)
                    reinterpret_cast<uint4*>(img)[i] = __ldcg(from + i);
            } else {
                (void)stage_groups<DT>(img, nullptr, p.x, nullptr, 0u, p.K, (uint32_t)warp, ge.ngroups, (uint32_t)kConsumers, lane);
            }
        } else {
            float ss = stage_groups<DT, !AL>(img, img + x_image_bytes(ge.ngroups) / 4u, p.x, p.x2, p.x_op, p.K, (uint32_t)warp, ge.ngroups, (uint32_t)kConsumers, lane);
            if (p.x_op == 1u) {
#pragma unroll
                for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                if (lane == 0) red[warp] = ss;
            }
        }
        consumer_sync();                                     // the image and the warps' partial sums of squares are in place
        if (tr) tr[2] = global_ns();
        RingPos pos{0, 0};
        consume<DT, AL>(rg, pos, ge, rows, p.K, smem_base(img), warp, lane, [&](uint32_t row) { return (uint32_t)(uintptr_t)row_ptr(p, cta_lo + row) & 15u; });
    }
    exchange_signal(p.xc);                                   // sharded models: this CTA's rows are on every peer
    if (tr) tr[3] = global_ns();
}

// ---- generic kernel: any alignment, byte loads, one warp per row --------------
template <int DT>
__device__ float generic_row(const uint8_t* r, const float* x, uint32_t K, int lane);

__device__ __forceinline__ float ldh(const uint8_t* p) { return half_to_float((uint32_t)p[0] | ((uint32_t)p[1] << 8)); }

template <> __device__ float generic_row<1>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    for (uint32_t b = lane; b < K / 32; b += 32) {
        const uint8_t* q = r + (size_t)b * 18;
        float s = 0.f;
        for (int j = 0; j < 16; ++j)
            s += (float)((int)(q[2 + j] & 15) - 8) * x[b * 32 + 2 * j] + (float)((int)(q[2 + j] >> 4) - 8) * x[b * 32 + 2 * j + 1];
        acc += s * ldh(q);
    }
    return acc;
}
template <> __device__ float generic_row<9>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    for (uint32_t b = lane; b < K / 32; b += 32) {
        const uint8_t* q = r + (size_t)b * 18;
        float s = 0.f;
        for (int j = 0; j < 16; ++j)
            s += (float)((int)(q[2 + j] & 15) - 8) * x[b * 32 + j] + (float)((int)(q[2 + j] >> 4) - 8) * x[b * 32 + 16 + j];
        acc += s * ldh(q);
    }
    return acc;
}
// TQ2: the reference's code-counting dot (quant.h:520-531): with lo / hi the two bits of a code,
// sum w x = d * (sum_{lo} x + 2 sum_{hi} x - sum x) per 128-block; one block per lane iteration.
template <> __device__ float generic_row<7>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    for (uint32_t b = lane; b < K / 128; b += 32) {
        const uint8_t* q = r + (size_t)b * 34;
        float lo = 0.f, hi = 0.f, all = 0.f;
        for (int j = 0; j < 32; ++j) {
            const uint32_t byte = q[2 + j];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float xv = x[b * 128 + 4 * j + t];
                const uint32_t c = (byte >> (2 * t)) & 3u;
                all += xv;
                if (c & 1u) lo += xv;
                if (c & 2u) hi += xv;
            }
        }
        acc += ldh(q) * (lo + 2.f * hi - all);
    }
    return acc;
}
template <> __device__ float generic_row<0>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    for (uint32_t b = lane; b < K / 32; b += 32) {
        const uint8_t* q = r + (size_t)b * 34;
        float s = 0.f;
        for (int j = 0; j < 32; ++j) s += (float)(int8_t)q[2 + j] * x[b * 32 + j];
        acc += s * ldh(q);
    }
    return acc;
}
template <> __device__ float generic_row<4>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    for (uint32_t b = lane; b < K / 32; b += 32) {
        const uint8_t* q = r + (size_t)b * 20;
        float s = 0.f, xs = 0.f;
        for (int j = 0; j < 16; ++j) {
            const float x0 = x[b * 32 + j], x1 = x[b * 32 + 16 + j];
            s += (float)(q[4 + j] & 15) * x0 + (float)(q[4 + j] >> 4) * x1;
            xs += x0 + x1;
        }
        acc += s * ldh(q) + xs * ldh(q + 2);
    }
    return acc;
}
template <> __device__ float generic_row<5>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    // one (super-block, sub-block) pair per lane iteration
    for (uint32_t u = lane; u < K / 32; u += 32) {
        const uint8_t* q = r + (size_t)(u >> 3) * 176;
        const uint32_t j = u & 7, g = j >> 1, hi = j & 1;
        const uint8_t* sc = q + 4;
        uint32_t s6, m6;
        if (j < 4) { s6 = sc[j] & 63u; m6 = sc[j + 4] & 63u; }
        else { s6 = (sc[j + 4] & 15u) | ((sc[j - 4] >> 6) << 4); m6 = (sc[j + 4] >> 4) | ((sc[j] >> 6) << 4); }
        float s = 0.f, xs = 0.f;
        for (int l = 0; l < 32; ++l) {
            const uint32_t nib = hi ? (q[48 + 32 * g + l] >> 4) : (q[48 + 32 * g + l] & 15u);
            const uint32_t code = nib + (((q[16 + l] >> j) & 1u) << 4);
            const float xv = x[(u >> 3) * 256 + j * 32 + l];
            s += (float)code * xv; xs += xv;
        }
        acc += ldh(q) * (float)s6 * s - ldh(q + 2) * (float)m6 * xs;
    }
    return acc;
}
template <> __device__ float generic_row<8>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    for (uint32_t u = lane; u < K / 32; u += 32) {          // one (super-block, sub-block) pair per lane iteration
        const uint8_t* q = r + (size_t)(u >> 3) * 144;
        const uint32_t j = u & 7, g = j >> 1, hi = j & 1;
        const uint8_t* sc = q + 4;
        uint32_t s6, m6;
        if (j < 4) { s6 = sc[j] & 63u; m6 = sc[j + 4] & 63u; }
        else { s6 = (sc[j + 4] & 15u) | ((sc[j - 4] >> 6) << 4); m6 = (sc[j + 4] >> 4) | ((sc[j] >> 6) << 4); }
        float s = 0.f, xs = 0.f;
        for (int l = 0; l < 32; ++l) {
            const uint32_t code = hi ? (q[16 + 32 * g + l] >> 4) : (q[16 + 32 * g + l] & 15u);
            const float xv = x[(u >> 3) * 256 + j * 32 + l];
            s += (float)code * xv; xs += xv;
        }
        acc += ldh(q) * (float)s6 * s - ldh(q + 2) * (float)m6 * xs;
    }
    return acc;
}
template <> __device__ float generic_row<6>(const uint8_t* r, const float* x, uint32_t K, int lane) {
    float acc = 0.f;
    // one 16-weight sub-block per lane iteration: sub = 8h + 2j + (l/16)
    for (uint32_t u = lane; u < K / 16; u += 32) {
        const uint8_t* q = r + (size_t)(u >> 4) * 210;
        const uint32_t sub = u & 15, h = sub >> 3, j = (sub >> 1) & 3, l0 = (sub & 1) * 16;
        float s = 0.f;
        for (uint32_t l = l0; l < l0 + 16; ++l) {
            const uint8_t qlb = q[64 * h + 32 * (j & 1) + l];
            const uint32_t lo = (j & 2) ? (qlb >> 4) : (qlb & 15u);
            const uint32_t hi2 = (q[128 + 32 * h + l] >> (2 * j)) & 3u;
            s += (float)((int)(lo | (hi2 << 4)) - 32) * x[(u >> 4) * 256 + 128 * h + 32 * j + l];
        }
        acc += ldh(q + 208) * (float)(int8_t)q[192 + sub] * s;
    }
    return acc;
}

template <int DT>
__global__ void __launch_bounds__(256) gemv_generic(const GemvParams p) {
    extern __shared__ __align__(16) float xs[];            // transformed x, only when a fused transform is requested
    __shared__ float red[8];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    exchange_wait(p.xc, p.status);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* x = p.x;
    if (p.x_op != 0u) {
        float inv = 1.f;
        if (p.x_op == 1u) {
            float ss = 0.f;
            for (uint32_t i = threadIdx.x; i < p.K; i += blockDim.x) { const float t = p.x[i]; ss = fmaf(t, t, ss); }
#pragma unroll
            for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) red[warp] = ss;
            __syncthreads();
            float tot = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
            inv = 1.0f / sqrtf(tot / (float)p.K + p.eps);
        }
        for (uint32_t i = threadIdx.x; i < p.K; i += blockDim.x) {
            const float t = p.x[i];
            xs[i] = p.x_op == 1u ? t * inv * p.x2[i] : t / (1.0f + expf(-t)) * p.x2[i];
        }
        __syncthreads();
        x = xs;
    }
    const uint32_t cta_lo = blockIdx.x * (blockDim.x >> 5), row = cta_lo + warp;
    if (row < p.N) {
        float v = generic_row<DT>(row_ptr(p, row), x, p.K, lane);
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const uint32_t e = y_index(p, row);
        if (lane == 0) {
            if (p.accumulate) v += p.y[e];
            p.y[e] = v;
            for (uint32_t q = 0; q < p.xc.npush; ++q) p.xc.peer_y[q][e] = v;         // a sharded model's peers
        }
    }
    exchange_signal(p.xc);
}

constexpr uint32_t kSmemLimit = 227 * 1024 - 512;        // dynamic part; the kernel also has a few static words
unsigned g_last_grid = 0;

template <int DT, bool AL>
bool launch_stream(const GemvParams& p, unsigned grid, size_t smem, cudaStream_t st) {
    static bool attr_set = false;
    static const bool pdl = [] { const char* e = std::getenv("TM_GEMV_PDL"); return !(e && *e == '0'); }();   // A/B knob: 0 launches without programmatic serialization
    if (!attr_set) {
        if (cudaFuncSetAttribute(gemv_stream<DT, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit) != cudaSuccess)
            return fail("gemv: cannot raise the dynamic shared memory limit");
        // every GEMV asks for the largest shared-memory carveout, so consecutive kernels share one SM configuration
        cudaFuncSetAttribute(gemv_stream<DT, AL>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(gemv_threads(DT)); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, gemv_stream<DT, AL>, p) != cudaSuccess) return check_launch("gemv_stream");
    g_last_grid = grid;
    note_launch();
    return true;
}

template <int DT> bool launch_generic_only(GemvParams p, cudaStream_t st);

// aligned: every row starts on a 16-byte boundary; even: on an even address.
template <int DT>
bool launch_dt(GemvParams p, bool aligned, bool even, cudaStream_t st, ShareCount* share) {
    p.ge = tile_geom(DT, p.K, aligned);
    const uint32_t fixed = x_smem(p.ge, aligned) + kRingBarBytes;
    if (!aligned) p.xq = nullptr;                           // such an image has two planes
    // A slot per producer at least: where x has four planes, some 29000 activations leave no room for the ring. Two would fit
    // twice as many, but above kMaxPlaneK x has always been multiplied in fp32, and two planes hold less: a small activation
    // beside a large one of its 32 keeps what is left of 15 bits.
    const bool held = !aligned || p.K <= kMaxPlaneK;
    if (even && held && fixed + p.ge.producers * p.ge.slot_bytes <= kSmemLimit) {
        const unsigned sms = (unsigned)device_sm_count();
        // as many CTAs as SMs, rows spread evenly: with one CTA per SM the longest range is the launch's time
        p.rows_per_cta = (p.N + sms - 1) / sms;
        const unsigned grid = (p.N + p.rows_per_cta - 1) / p.rows_per_cta;
        const unsigned items = (p.rows_per_cta + kTileRows - 1) / kTileRows * p.ge.nchunks;
        unsigned S = (kSmemLimit - fixed) / p.ge.slot_bytes;
        if (S > (unsigned)kRingSlots) S = kRingSlots;
        if (S > items) S = items;
        p.slots = S;
        const size_t smem = fixed + (size_t)S * p.ge.slot_bytes;
        if (p.share && aligned)                             // CTA b makes groups b, b + grid, ...: a part each, while there are groups
            return share->launch(p.ge.ngroups < grid ? p.ge.ngroups : grid, [&](unsigned want) {
                p.share_want = want;
                return launch_stream<DT, true>(p, grid, smem, st);
            });
        return aligned ? launch_stream<DT, true>(p, grid, smem, st) : launch_stream<DT, false>(p, grid, smem, st);
    }
    return launch_generic_only<DT>(p, st);
}

template <int DT>
bool launch_generic_only(GemvParams p, cudaStream_t st) {
    p.xq = nullptr;                                         // the plain kernel reads the fp32 x
    const unsigned rows_per_cta = 8;
    const size_t xsmem = p.x_op ? (size_t)p.K * 4 : 0;
    if (xsmem > 48 * 1024) {
        static bool attr = false;
        if (!attr && cudaFuncSetAttribute(gemv_generic<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
            return fail("gemv: cannot raise the dynamic shared memory limit");
        attr = true;
        if (xsmem > 200 * 1024) return fail("gemv: K=%u is too long for the unaligned fused form", p.K);
    }
    gemv_generic<DT><<<(p.N + rows_per_cta - 1) / rows_per_cta, rows_per_cta * 32, xsmem, st>>>(p);
    g_last_grid = (p.N + rows_per_cta - 1) / rows_per_cta;
    note_launch();
    return check_launch("gemv_generic");
}

bool launch_any(const GemvParams& p, unsigned dtype, bool aligned, bool even, cudaStream_t st, ShareCount* share) {
    switch (dtype) {
        case DT_Q8_0: return launch_dt<0>(p, aligned, even, st, share);
        case DT_Q4_0: return launch_dt<1>(p, aligned, even, st, share);
        case DT_Q4_1: return launch_dt<4>(p, aligned, even, st, share);
        case DT_Q5_K: return launch_dt<5>(p, aligned, even, st, share);
        case DT_Q4_K: return launch_dt<8>(p, aligned, even, st, share);
        case DT_GGUF_Q4_0: return launch_dt<9>(p, aligned, even, st, share);
        default: return launch_dt<6>(p, aligned, even, st, share);
    }
}
}  // namespace

unsigned last_gemv_grid() { return g_last_grid; }

bool launch_gemv(const float* x, const uint8_t* W, float* y, unsigned N, unsigned K, unsigned dtype,
                 const SegTable& seg, cudaStream_t st, const GemvFuse* fuse) {
    const unsigned be = block_elems(dtype);
    if (!be || dtype == DT_F16) return fail("gemv: dtype %u is not a block format", dtype);
    if (!x || !W || !y) return fail("gemv: null pointer");
    if (N == 0) return true;
    if (K == 0 || K % be) return fail("gemv: K=%u is not a multiple of %u", K, be);
    if (seg.nseg == 0 || seg.nseg > (unsigned)kMaxSeg) return fail("gemv: %u segments (1..%d supported)", seg.nseg, kMaxSeg);
    if (seg.row_end[seg.nseg - 1] != N) return fail("gemv: segment rows do not add up to N");
    if ((uintptr_t)x % 16) return fail("gemv: x must be 16-byte aligned");
    GemvParams p;
    p.W = W; p.x = x; p.y = y; p.N = N; p.K = K;
    p.row_bytes = (K / be) * block_bytes(dtype);
    p.seg = seg; p.status = device_status_word(); p.trace = device_trace();
    p.x2 = nullptr; p.eps = 0.f; p.x_op = 0; p.accumulate = 0;
    p.xc = Exchange{};
    p.xq = nullptr; p.share = nullptr; p.share_ctr = nullptr; p.share_want = 0; p.share_ns = 0;
    if (fuse && fuse->xchg) p.xc = *fuse->xchg;
    if (p.xc.npush > (unsigned)kMaxPeers || (p.xc.nwait && (!p.xc.wait_ctrs || !p.xc.wait_ctas || !p.xc.epoch)))
        return fail("gemv: incomplete peer exchange description");
    p.x_ns = 2ull * kWaitLimitNs + p.xc.nwait * p.xc.limit_ns;      // the peers' limits, one after another, and what the kernel waits for itself
    if (fuse) {
        if (fuse->x_op > 2 || (fuse->x_op != 0 && (!fuse->x2 || (uintptr_t)fuse->x2 % 16))) return fail("gemv: bad fused x transform");
        p.x2 = fuse->x2; p.eps = fuse->eps; p.x_op = fuse->x_op; p.accumulate = fuse->accumulate ? 1u : 0u;
        if (fuse->xq) {
            if ((uintptr_t)fuse->xq % 16) return fail("gemv: the staged x image must be 16-byte aligned");
            p.xq = fuse->xq;
        }
        // TM_GEMV_SHARE_WAIT_US: 0 has every CTA stage x for itself
        static const unsigned long long share_ns = [] { const char* e = std::getenv("TM_GEMV_SHARE_WAIT_US"); return e && *e ? 1000ull * std::strtoul(e, nullptr, 10) : 200000ull; }();
        if (fuse->share && fuse->x_op == 0) { p.share_ns = share_ns; p.share = fuse->share; p.share_ctr = fuse->share_count->parts; }
    }
    bool aligned = ((uintptr_t)W % 16 == 0) && (p.row_bytes % 16 == 0), even = (uintptr_t)W % 2 == 0;
    for (unsigned s = 0; s < seg.nseg; ++s) { aligned = aligned && (seg.woff[s] % 16 == 0); even = even && (seg.woff[s] % 2 == 0); }
    if (dtype == DT_TQ2) {                                  // ternary rows: the plain kernel (no streaming lane is built for them)
        p.xq = nullptr;
        return launch_generic_only<7>(p, st);
    }
    return launch_any(p, dtype, aligned, even, st, fuse ? fuse->share_count : nullptr);
}

size_t xq_bytes(unsigned K, unsigned dtype) {
    if (!block_elems(dtype) || dtype == DT_TQ2) return 0;
    return (size_t)kXqHeaderWords * 4 + (size_t)((K + 255u) / 256u) * kXGroupWords * 4u;
}

namespace {
template <int CDT>
bool launch_xprep_dt(uint32_t* out, const float* x, const float* x2, unsigned x_op, float eps, unsigned K, const Exchange& xc, cudaStream_t st) {
    const unsigned ngroups = (K + 255u) / 256u;
    // RMSNorm sums over the whole vector: one CTA of 16 warps. Otherwise four groups per CTA.
    const unsigned threads = x_op == 1u ? 512u : 128u, grid = x_op == 1u ? 1u : (ngroups + 3u) / 4u;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = 0; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, xprep_kernel<CDT>, out, x, x2, (uint32_t)x_op, eps, (uint32_t)K, xc, device_status_word()) != cudaSuccess)
        return check_launch("xprep");
    note_launch();
    return true;
}
}  // namespace

bool launch_xprep(uint32_t* out, const float* x, const float* x2, unsigned x_op, float eps, unsigned K, unsigned dtype,
                  const Exchange* xchg, cudaStream_t st) {
    if (!out || !x || (uintptr_t)out % 16 || (uintptr_t)x % 16 || x_op > 2 || (x_op && (!x2 || (uintptr_t)x2 % 16)))
        return fail("xprep: bad arguments");
    const unsigned be = block_elems(dtype);
    if (!be || dtype == DT_F16 || K == 0 || K % be) return fail("xprep: K=%u is not whole blocks of dtype %u", K, dtype);
    const Exchange xc = xchg ? *xchg : Exchange{};
    switch (dtype) {
        case DT_Q8_0: return launch_xprep_dt<0>(out, x, x2, x_op, eps, K, xc, st);
        case DT_Q4_0: return launch_xprep_dt<1>(out, x, x2, x_op, eps, K, xc, st);
        case DT_Q4_1: return launch_xprep_dt<4>(out, x, x2, x_op, eps, K, xc, st);
        case DT_Q5_K: return launch_xprep_dt<5>(out, x, x2, x_op, eps, K, xc, st);
        case DT_Q4_K: return launch_xprep_dt<8>(out, x, x2, x_op, eps, K, xc, st);
        case DT_GGUF_Q4_0: return launch_xprep_dt<9>(out, x, x2, x_op, eps, K, xc, st);
        default: return launch_xprep_dt<6>(out, x, x2, x_op, eps, K, xc, st);
    }
}

}  // namespace tmc
