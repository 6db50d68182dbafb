// gemv_tile.cuh — the pieces of the streaming GEMV that its kernels share: bulk copies on mbarriers, the staging of x,
// and the geometry of a CTA's tile stream.
//
// A CTA's rows are cut into tiles of 16 (the MMA's row count) and a row's groups of 256 weights into chunks of kw
// groups. An item of the stream is one chunk of one tile: 16 bulk copies, one per row, into one slot of a shared-memory
// ring, at a row stride that keeps the lanes' loads free of bank conflicts. Items come in the order tile group, chunk,
// tile of the group; a tile group is rw = 16 / kw tiles, one for each team of kw consumer warps, warp k of a team taking
// the k-th group of the chunk. A slot goes round three mbarriers: full (its bytes have landed), done (every consumer
// warp is through with the item, its team having left one partial sum per row, group and quarter beside the slot), spare
// (the reducer warps have added them up and stored finished rows: the producers may refill). So no warp that multiplies
// waits for another one that does. Every role takes every item in order, also the warps of the teams whose item it is
// not: a phase of a slot's barrier is then never more than one away from what a warp waits for, which is what one
// parity bit can tell.
// The partial sums are added in an order that depends on K only (row_sum), so a row's bits do not depend on how many
// rows the launch has, on the split, or on how the row was reached.
#pragma once

#include "common.cuh"
#include "gemv_lanes.cuh"
#include "bulk.cuh"

namespace tmc {

constexpr int kConsumers = 16;                              // warps that multiply
constexpr int kProducers = 4;                               // warps that issue the row copies (two to four of them do)
// Warps that add a tile's partial sums and store its rows. Formats that are cheap to multiply go through more tiles per
// microsecond and want four (Q8_0 32000 x 2048 13.0 -> 12.8 us, Q4_0 28672 x 4096 13.4 -> 13.1, a token of 8B shapes 1 %); the K-quants
// lose more issue slots to the two extra warps than they gain (Q6_K 128256 x 4096 74.4 -> 76.7).
__host__ __device__ constexpr int reducers(int dt) { return dt == 5 || dt == 6 || dt == 8 ? 2 : 4; }
constexpr int gemv_threads(int dt) { return 32 * (kConsumers + kProducers + reducers(dt)); }
constexpr int kTileRows = 16;
constexpr int kRingSlots = 16;                              // most slots of a ring (its barriers have fixed places)

// Geometry of a tile stream that does not depend on the rows.
struct TileGeom {
    uint32_t kw, rw, nchunks, ngroups;
    uint32_t chunk_bytes;                                   // bytes of a full chunk of one row
    uint32_t stride;                                        // bytes between the rows of an item in shared memory
    uint32_t prow;                                          // floats between two rows of an item's partial sums
    uint32_t slot_bytes;                                    // the item's bytes and its partial sums
    uint32_t producers;                                     // producer warps at work
};

inline __host__ __device__ uint32_t group_bytes(unsigned dt) {
    switch (dt) { case 0: return 272; case 1: case 8: case 9: return 144; case 4: return 160; case 5: return 176; default: return 210; }
}
// Stage stride: 16-byte rows an odd number of 16-byte units apart put the eight rows that a load touches into eight
// different bank groups (Q4_1's 8-byte loads want an odd number of 32-byte units).
inline __host__ __device__ uint32_t stage_stride(unsigned dt, uint32_t chunk_bytes, bool aligned) {
    const uint32_t unit = dt == 4 ? 32u : 16u;
    uint32_t u = (chunk_bytes + (aligned ? 0u : 16u) + unit - 1u) / unit;
    return (u | 1u) * unit;
}
// kw: a row in one chunk while an item stays near 40 KB (deep enough a ring for the DRAM latency) and there are warps for
// it; longer rows in whole steps of eight groups, eight or sixteen at a time, whichever leaves fewer warps idle in the
// last chunk. Whole steps are also what keeps the chunks of Q6_K rows aligned (eight super-blocks are 1680 bytes).
inline __host__ __device__ TileGeom tile_geom(unsigned dt, uint32_t K, bool aligned) {
    TileGeom g;
    const uint32_t gb = group_bytes(dt);
    uint32_t most = 41984u / (16u * gb);
    if (most > 16u) most = 16u;
    g.ngroups = (K + 255u) / 256u;
    if (g.ngroups <= most) g.kw = g.ngroups;
    else g.kw = most == 16u && (g.ngroups & 15u) - 1u >= 8u ? 16u : 8u;
    g.nchunks = (g.ngroups + g.kw - 1u) / g.kw;
    g.rw = 16u / g.kw;
    g.chunk_bytes = g.kw * gb;
    g.stride = stage_stride(dt, g.chunk_bytes, aligned);
    g.prow = ((g.kw + 7u) & ~7u) * 4u + 4u;                 // four quarters per group of whole steps; the pad spreads the rows over the banks
    // A warp's sixteen row copies take it 0.6-0.7 us: two warps keep up with the HBM rate from 2 KB copies on, shorter ones
    // want a third (Q6_K 128256 x 4096, 1680-byte copies: 81.9 -> 75.0 us; Q4_1 32000 x 2048, 1280: 10.8 -> 9.7), which
    // only gets in the way of long ones (Q4_0 28672 x 4096, 2304: 13.1 -> 14.1). Copies around a kilobyte and below want a
    // fourth (102687 x 1024 Q4_0, 576 bytes: 22.0 -> 19.5; 81669 x 1792, 1008: 21.0 -> 20.0; Q8_0 54564 x 256, 272: 12.3 -> 10.8).
    g.producers = g.chunk_bytes < 1200u ? 4u : g.chunk_bytes < 2048u ? 3u : 2u;
    g.slot_bytes = (kTileRows * (g.stride + 4u * g.prow) + 127u) & ~127u;
    return g;
}
inline __host__ __device__ uint32_t x_image_bytes(uint32_t ngroups) { return ((ngroups + 1u) * (uint32_t)kXGroupWords * 4u + 127u) & ~127u; }   // and a group of zeros

__device__ __forceinline__ void st_f(uint32_t p, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory"); }
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kConsumers * 32) : "memory"); }

// The sums of two rows' partials of an item (n <= kw groups; pa, pb: the rows' addresses, at this lane's quarter), by four
// neighbouring lanes (every lane of the warp calls), added to a and b. Fixed order: within a step of eight groups
// ((0+4)+(2+6))+((1+5)+(3+7)) for every quarter, then the quarters (0+2)+(1+3), then the steps in order; items are whole
// steps or whole rows, so that is the order over the row.
__device__ __forceinline__ void row_sum(SPtr pa, SPtr pb, uint32_t n, float& a, float& b, bool first) {
    for (uint32_t s = 0; s < n; s += 8, pa += 128u, pb += 128u) {
        float q[8], r[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) { q[k] = __uint_as_float(ld4(pa + 16u * k)); r[k] = __uint_as_float(ld4(pb + 16u * k)); }   // places for whole steps are there
        if (s + 8 > n) {
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) { q[k] = s + k < n ? q[k] : 0.f; r[k] = s + k < n ? r[k] : 0.f; }
        }
        float u = ((q[0] + q[4]) + (q[2] + q[6])) + ((q[1] + q[5]) + (q[3] + q[7]));
        float v = ((r[0] + r[4]) + (r[2] + r[6])) + ((r[1] + r[5]) + (r[3] + r[7]));
        u += __shfl_xor_sync(0xffffffffu, u, 2); v += __shfl_xor_sync(0xffffffffu, v, 2);
        u += __shfl_xor_sync(0xffffffffu, u, 1); v += __shfl_xor_sync(0xffffffffu, v, 1);
        a = first && s == 0 ? u : a + u;
        b = first && s == 0 ? v : b + v;
    }
}

// ---- staging of x: block floating point planes in the MMA's operand layout -------------------------------------------
// Eight lanes per 32-block, four activations (one float4) per lane: the block maximum and the block sum come from three
// shuffle stages, the plane bytes leave as packed stores. A warp stages eight blocks (one group) per pass; it takes
// groups g_first, g_first + g_step, ... below g_end. `units` is shared memory (a CTA staging for itself) or global
// memory (staging once for every CTA of a later launch). Blocks past K inside the last group are staged as zeros.
// FINE: two more planes, into an image of their own at `fine`. Returns this lane's share of sum(x^2) for x_op 1 (RMSNorm: x * w is staged, the factor rsqrt(mean(x^2) + eps) is one
// number for the whole vector and multiplies the finished row sums instead); x_op 2 stages silu(x) * x2.
template <int DT, bool FINE = false>
__device__ __forceinline__ float stage_groups(uint32_t* units, uint32_t* fine, const float* x, const float* x2, uint32_t x_op, uint32_t K,
                                              uint32_t g_first, uint32_t g_end, uint32_t g_step, int lane) {
    using L = Lane<DT>;
    constexpr int B = 2;
    const uint32_t nblk = K / 32, li = lane & 7u, sub = lane >> 3;
    const float4* xg4 = reinterpret_cast<const float4*>(x);
    const float4* x24 = reinterpret_cast<const float4*>(x2);
    float ss = 0.f;
    // The loads of the next group are issued before the current group is quantized: a warp's passes are
    // otherwise a chain of L2 latencies.
    float4 nv[B], nw[B];
    auto fetch = [&](uint32_t g) {
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const uint32_t b = g * (4 * B) + 4 * j + sub;
            const bool in = g < g_end && b < nblk;
            nv[j] = in ? __ldcg(xg4 + b * 8 + li) : make_float4(0.f, 0.f, 0.f, 0.f);
            nw[j] = (in && x_op != 0u) ? __ldcg(x24 + b * 8 + li) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(g_first);
    for (uint32_t g = g_first; g < g_end; g += g_step) {
        const uint32_t b0 = g * (4 * B);
        float4 v[B];
        float s16[B], s32[B];
        uint32_t am[B];                                      // max |x| as bits: they order like the magnitudes, infinity and NaN above everything finite
        float4 w2s[B];
#pragma unroll
        for (int j = 0; j < B; ++j) { v[j] = nv[j]; w2s[j] = nw[j]; }
        fetch(g + g_step);
#pragma unroll
        for (int j = 0; j < B; ++j) {
            if (x_op == 1u) {
                const float4 w2 = w2s[j];
                ss = fmaf(v[j].x, v[j].x, ss); ss = fmaf(v[j].y, v[j].y, ss); ss = fmaf(v[j].z, v[j].z, ss); ss = fmaf(v[j].w, v[j].w, ss);
                v[j].x *= w2.x; v[j].y *= w2.y; v[j].z *= w2.z; v[j].w *= w2.w;
            } else if (x_op == 2u) {
                // silu(x) * up with the hardware exponential and reciprocal: relative error 2^-21, inside what the two
                // fixed-point planes that follow keep; four planes keep more
                const float4 w2 = w2s[j];
                if constexpr (FINE) {
                    v[j].x = v[j].x / (1.0f + expf(-v[j].x)) * w2.x; v[j].y = v[j].y / (1.0f + expf(-v[j].y)) * w2.y;
                    v[j].z = v[j].z / (1.0f + expf(-v[j].z)) * w2.z; v[j].w = v[j].w / (1.0f + expf(-v[j].w)) * w2.w;
                } else {
                    v[j].x = __fdividef(v[j].x, 1.0f + __expf(-v[j].x)) * w2.x; v[j].y = __fdividef(v[j].y, 1.0f + __expf(-v[j].y)) * w2.y;
                    v[j].z = __fdividef(v[j].z, 1.0f + __expf(-v[j].z)) * w2.z; v[j].w = __fdividef(v[j].w, 1.0f + __expf(-v[j].w)) * w2.w;
                }
            }
            am[j] = max(max(__float_as_uint(fabsf(v[j].x)), __float_as_uint(fabsf(v[j].y))), max(__float_as_uint(fabsf(v[j].z)), __float_as_uint(fabsf(v[j].w))));
            s32[j] = (v[j].x + v[j].y) + (v[j].z + v[j].w);
        }
#pragma unroll
        for (int o = 1; o <= 4; o <<= 1)
#pragma unroll
            for (int j = 0; j < B; ++j) {
                am[j] = max(am[j], __shfl_xor_sync(0xffffffffu, am[j], o));
                if (L::NEEDS_SUMS) { s32[j] += __shfl_xor_sync(0xffffffffu, s32[j], o); if (o == 2) s16[j] = s32[j]; }
            }
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const uint32_t b = b0 + 4 * j + sub;
            float inv;
            const float amax = __uint_as_float(am[j]), sc = block_scale(amax, !(amax <= 3.0e38f), inv);
            uint32_t q1, q2;
            quantize_quad(v[j].x, v[j].y, v[j].z, v[j].w, inv, q1, q2);
            L::store_quad(units, b * 32 + 4 * li, 0, q1);
            L::store_quad(units, b * 32 + 4 * li, 1, q2);
            if constexpr (FINE) {
                quantize_rest(v[j].x, v[j].y, v[j].z, v[j].w, inv, q1, q2);
                L::store_quad(fine, b * 32 + 4 * li, 0, q1);
                L::store_quad(fine, b * 32 + 4 * li, 1, q2);
            }
            L::scalars(units, b, (int)(4 * li), (int)li, sc, 0.f, s16[j], s32[j]);
        }
    }
    return ss;
}

// ---- the ring and its three roles ------------------------------------------------------------------------------------
// What the waits of a CTA's ring share (in shared memory). Producers and reducers may have to wait for as long as the consumers
// wait for x: for the preceding kernel, whose time does not count, and for the peers of a sharded model. So a wait whose
// usual limit has passed first lets the preceding kernel end and then gives the rest `ns`. (Looked at only then: most waits
// come here for a moment, and anything done on the way in is paid for by every slot.) One that runs out says so in the
// status word.
struct Patience {
    int gone;                                               // a wait ran out: nobody waits as long again
    int* status;
    unsigned long long ns;
};
static __device__ __noinline__ bool ring_wait_slow(uint32_t bar, uint32_t parity, volatile Patience* pt) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = global_ns(), limit = kWaitLimitNs;
    for (bool last = false;;) {
        for (int i = 0; i < 64; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (pt->gone) break;
        if (global_ns() - t0 <= limit) continue;
        if (last) break;
        last = true;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        t0 = global_ns();
        limit = pt->ns;
    }
    pt->gone = 1;
    *(volatile int*)pt->status = 1;
    return false;
}
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity, Patience* pt) { return mbar_test(bar, parity) || ring_wait_slow(bar, parity, pt); }

struct Ring {
    uint32_t at;                                            // shared-memory address of slot 0
    uint32_t bars;                                          // full[kRingSlots], done[kRingSlots], spare[kRingSlots]
    uint32_t slots, slot_bytes;
    Patience* patience;
    __device__ __forceinline__ uint32_t full(uint32_t s) const { return bars + 8u * s; }
    __device__ __forceinline__ uint32_t done(uint32_t s) const { return bars + 8u * (kRingSlots + s); }
    __device__ __forceinline__ uint32_t spare(uint32_t s) const { return bars + 8u * (2u * kRingSlots + s); }
    __device__ __forceinline__ void init(uint32_t reds) const {      // one thread, before anybody waits
        for (uint32_t s = 0; s < slots; ++s) { mbar_init(full(s), 1); mbar_init(done(s), kConsumers); mbar_init(spare(s), reds); }
    }
};
constexpr uint32_t kRingBarBytes = 3 * kRingSlots * 8;
struct RingPos {                                            // a role's place in the ring: slot and the parity it waits for there
    uint32_t slot, par;
    __device__ __forceinline__ void next(uint32_t slots) { if (++slot == slots) { slot = 0; par ^= 1u; } }
};
// The items of `tiles` tiles in stream order: f(tile, chunk, team).
template <typename F> __device__ __forceinline__ void for_items(const TileGeom& ge, uint32_t tiles, F f) {
    for (uint32_t tg = 0; tg < tiles; tg += ge.rw) {
        const uint32_t rr = min(ge.rw, tiles - tg);
        for (uint32_t c = 0; c < ge.nchunks; ++c)
            for (uint32_t r = 0; r < rr; ++r) f(tg + r, c, r);
    }
}

// Producer `mine`: the row copies of every ge.producers-th item. pos starts at parity 1 (the first pass over the ring finds
// every slot free). rows: how many there are; src(row): its address. The ring has as many slots as producers at least, so
// a producer that waits for item i's slot has seen item i - slots - producers freed, and with it everything before (a
// reducer frees in order and all arrive for every item): the phase it waits for is the next one.
template <bool AL, typename Src>
__device__ __forceinline__ bool produce(const Ring& rg, RingPos& pos, const TileGeom& ge, uint32_t rows, uint32_t row_bytes,
                                        uint32_t mine, int lane, Src src_of) {
    bool ok = true;
    uint32_t turn = 0;
    for_items(ge, (rows + kTileRows - 1) / kTileRows, [&](uint32_t tile, uint32_t c, uint32_t) {
        if (turn == mine && ok) {
            if (!__all_sync(0xffffffffu, ring_wait(rg.spare(pos.slot), pos.par, rg.patience))) {
                ok = false;
            } else {
                const uint32_t row = tile * kTileRows + (uint32_t)lane, off = c * ge.chunk_bytes, len = min(ge.chunk_bytes, row_bytes - off);
                const bool live = lane < kTileRows && row < rows;
                const uint8_t* src = live ? src_of(row) + off : nullptr;
                uint32_t bytes = live ? len : 0u, total;
                if constexpr (AL) {
                    total = (uint32_t)__popc(__ballot_sync(0xffffffffu, live)) * len;
                } else {                                     // from the 16-byte boundary below the row to the one above its end
                    const uint32_t mis = (uint32_t)(uintptr_t)src & 15u;
                    src -= mis;
                    bytes = live ? (bytes + mis + 15u) & ~15u : 0u;
                    total = __reduce_add_sync(0xffffffffu, bytes);
                }
                if (lane == 0) mbar_expect_tx(rg.full(pos.slot), total);
                __syncwarp();
                if (live) bulk_g2s(rg.at + pos.slot * rg.slot_bytes + (uint32_t)lane * ge.stride, src, bytes, rg.full(pos.slot));
            }
        }
        if (++turn == ge.producers) turn = 0;
        pos.next(rg.slots);
    });
    return ok;
}
// After a wait that ran out: copies may still be in flight into this CTA's shared memory; a last bounded chance to land.
__device__ __forceinline__ void drain(const Ring& rg) {
    volatile int* gone = &rg.patience->gone;
    *gone = 0;
    for (uint32_t s = 0; s < rg.slots; ++s) (void)mbar_wait(rg.full(s), 0, gone, 50000000ull), (void)mbar_wait(rg.full(s), 1, gone, 50000000ull);
}

// Consumer warp: multiplies its groups by x (image at shared address img). AL = false: rows on any even address; mis(row)
// gives the low four bits of a row's first byte, and x has four planes (a second image behind the first). The loop is short of issue slots on the 4-bit formats (41 weights per clock and SM at the HBM
// rate), so what it needs is in registers and its control is warp-uniform: a wait, the group, an arrival.
// ONE: a row is one chunk, so a warp multiplies by the same group throughout and keeps it in registers.
template <int DT, bool AL, bool ONE, typename Mis>
__device__ __forceinline__ void consume_items(const Ring& rg, RingPos& pos, const TileGeom& ge, uint32_t rows, uint32_t K, uint32_t img, int warp, int lane, Mis mis) {
    using L = Lane<DT>;
    const uint32_t g = (uint32_t)lane >> 2, t = (uint32_t)lane & 3u, kw = ge.kw, team = (uint32_t)warp / kw, wk = (uint32_t)warp % kw;
    const uint32_t ngroups = ge.ngroups, nchunks = ONE ? 1u : ge.nchunks, rw = ge.rw, stride8 = 8u * ge.stride, prow8 = 32u * ge.prow;
    const bool column = (g >> 1) == t;                      // this thread's B column belongs to its own k range
    const uint32_t xb0 = img + (column ? wk * kXGroupWords + 4u * g : ngroups * kXGroupWords) * 4u, xb_step = column ? kw * kXGroupWords * 4u : 0u;
    const uint32_t fine_off = column ? x_image_bytes(ngroups) : 0u;        // AL = false: the second pair of planes
    const uint32_t xf0 = img + (wk * kXGroupWords + 128u + 8u * t) * 4u;
    const uint32_t short_last = L::LANE_UNITS == 2 && (K & 255u) ? ngroups - 1u : ~0u;     // the group with missing blocks
    const uint32_t src0 = rg.at + g * ge.stride + wk * (uint32_t)L::GB + quarter_off<DT>(t);
    const uint32_t dst0 = rg.at + kTileRows * ge.stride + 4u * (g * ge.prow + 4u * wk + t);
    const uint32_t tiles = (rows + kTileRows - 1) / kTileRows;
    XRegs x;
    if (ONE) load_x<DT, !AL>(x, xb0, xf0);
    uint32_t tg = 0, c = 0, r = 0, gi = wk, rr = min(rw, tiles);
#pragma unroll 1
    for (uint32_t left = tiles * nchunks; left; --left) {
        (void)ring_wait(rg.full(pos.slot), pos.par, rg.patience);     // when it ran out, what is multiplied does not matter
        if (r == team && (ONE || gi < ngroups)) {
            const uint32_t at = pos.slot * rg.slot_bytes;
            uint32_t r0 = src0 + at, r1 = r0 + stride8;
            if constexpr (!AL) {
                const uint32_t row = (tg + r) * kTileRows + g, off = c * ge.chunk_bytes;
                r0 += (mis(min(row, rows - 1u)) + off) & 15u;
                r1 += (mis(min(row + 8u, rows - 1u)) + off) & 15u;
            }
            int nvalid = 2;
            if (gi == short_last) { const uint32_t nblk = (K & 255u) / 32u; nvalid = (int)min(2u, max(nblk, 2u * t) - 2u * t); }
            if (!ONE) load_x<DT, !AL>(x, xb0 + c * xb_step, xf0 + c * (kw * kXGroupWords * 4u));
            float acc0, acc1;
            group_dot<DT, AL, !AL>(r0, r1, x, xb0 + c * xb_step, xb0 + c * xb_step + fine_off, (int)t, nvalid, acc0, acc1);
            st_f(dst0 + at, acc0);
            st_f(dst0 + at + prow8, acc1);
        }
        __syncwarp();                                       // every lane is done with this slot
        mbar_arrive_if(rg.done(pos.slot), lane == 0);
        pos.next(rg.slots);
        if (++r == rr) {
            r = 0;
            if (ONE) {
                tg += rw; rr = min(rw, tiles - tg);
            } else {
                gi += kw;
                if (++c == nchunks) { c = 0; gi = wk; tg += rw; rr = min(rw, tiles - tg); }
            }
        }
    }
}
template <int DT, bool AL, typename Mis>
__device__ __forceinline__ void consume(const Ring& rg, RingPos& pos, const TileGeom& ge, uint32_t rows, uint32_t K, uint32_t img, int warp, int lane, Mis mis) {
    if (ge.nchunks == 1u) consume_items<DT, AL, true>(rg, pos, ge, rows, K, img, warp, lane, mis);
    else consume_items<DT, AL, false>(rg, pos, ge, rows, K, img, warp, lane, mis);
}

// Reducer `mine` of R: tiles mine, mine + R, ... (R >= 2, the tiles that a long row's chunks alternate between.) What a reducer does per tile is a chain of latencies (wait,
// loads, sums, shuffles, store), and it was the slowest role when both took half of every tile (750 clocks per item;
// Q4_0 28672 x 4096 13.9 -> 13.1 us, 4096 x 4096 4.6 -> 4.3).
// store(row, sum) is called by one lane per finished row. ready() is called once, after the first item is through the
// consumers.
template <uint32_t R, typename Ready, typename Store>
__device__ __forceinline__ void reduce(const Ring& rg, RingPos& pos, const TileGeom& ge, uint32_t rows, uint32_t mine, int lane, Ready ready, Store store) {
    const uint32_t g = (uint32_t)lane >> 2, t = (uint32_t)lane & 3u, prow = 4u * ge.prow, part0 = rg.at + kTileRows * ge.stride + prow * g + 4u * t;
    const uint32_t kw = ge.kw, ngroups = ge.ngroups, last = ge.nchunks - 1u;
    float v0 = 0.f, v1 = 0.f;                               // rows g and g + 8 of the tile in hand
    bool first = true;
    for_items(ge, (rows + kTileRows - 1) / kTileRows, [&](uint32_t tile, uint32_t c, uint32_t) {
        (void)ring_wait(rg.done(pos.slot), pos.par, rg.patience);
        if (first) { first = false; ready(); }
        if (tile % R == mine) {
            const uint32_t part = part0 + pos.slot * rg.slot_bytes, n = min(kw, ngroups - c * kw);
            row_sum(part, part + 8u * prow, n, v0, v1, c == 0u);
            __syncwarp();
            mbar_arrive_if(rg.spare(pos.slot), lane == 0);
            const uint32_t row = tile * kTileRows + g + (t << 3);      // lanes 0 and 1 of a row's four have rows g and g + 8
            if (c == last && t < 2u && row < rows) store(row, t ? v1 : v0);
        } else {
            mbar_arrive_if(rg.spare(pos.slot), lane == 0);  // in order and for every item, so that a freed slot means that all before it are free
        }
        pos.next(rg.slots);
    });
}

}  // namespace tmc
