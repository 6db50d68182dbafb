// gemm_blocks.cu — C[M x N] = A[M x K] W^T straight from the serialized blocks: no fp16 copy of the weights in memory.
//
// The two-launch form (gemm.cu: dequantize everything to fp16, then a TMA-fed GEMM) moves 4.5 + 16 + 16 bits per weight
// for a 4-bit type where the contraction needs 4.5, and pays a launch that nothing overlaps; with few tokens that was
// nearly all of the call. Here a weight goes
//     serialized bytes -> shared memory (16-byte copies)  -> registers -> fp16 pairs (gemm_codes.cuh) -> TMEM (tcgen05.st)
// and tcgen05.mma takes its A operand (128 weight rows) from TMEM, B (the tokens, fp16) from shared memory. Converting
// into TMEM instead of a swizzled shared-memory tile saves the shared-memory port both the store and the MMA's read of
// the 16 KB that 64 columns of K take, which together cost as long as the conversion itself; and a thread owns a row, the
// shape in which blocks are cheapest to decode.
// Bound: few tokens, the chain of latencies (first bytes 4 us after the launch, then about 750 clocks of conversion per
// group, the exchange); many rows, the conversion; 256 tokens and up, the MMAs. 17 tokens x 4096 x 4096, caches cold:
// Q4_0 33.8 -> 16.4 us, Q6_K 37.9 -> 20.5; 256 tokens Q4_0 35.8 -> 25.6, Q8_0 56 -> 25.6, Q5_K 85 -> 36; 17 x 32000 x 4096
// Q4_0 128 -> 46.
//
// K goes in groups of 256 weights = four stages of 64; the four sets of converter warps own one stage of every group each.
//   warps 0-15   converters: warp w takes TMEM lanes 32 (w % 4) .. + 32 (= rows) and stage w / 4 of every group
//   warps 16-19  epilogue
//   warp 20      MMA issuer (and TMEM allocation): two stages per step
//   warp 21      producer of token tiles, two stages per tensor copy
//   warps 22, 23 producers of raw groups, 16 bytes per lane and copy, neighbouring lanes along a row; where a CTA has one
//                tile only, the epilogue warps help until there is something to store. (A tensor copy brought 128 rows of
//                144 bytes in 1.0-1.5 us, slower than they are converted; requesting from the converter warps cost them
//                as many instructions as the conversion.)
// TMEM: accumulator(s) from column 0, fp16 weight slots (two stages, 64 columns) from the top down.
//
// Few tokens (their part of K fits beside the raw ring): the converters, who would wait for the first raw group, round
// the tokens into shared memory themselves, and the call is one launch. Otherwise a launch before this one writes them to
// the scratch buffer, already in the order of k_of.
//
// Few tiles: a cluster of up to eight CTAs shares one tile, each a part of K; the partial tiles are exchanged through
// distributed shared memory and summed in CTA order, so the result does not depend on timing.
#include "common.cuh"
#include "bulk.cuh"
#include "gemm.h"
#include "gemm_codes.cuh"

#include <cstdlib>

#include <cuda.h>
#include <cuda_fp16.h>

namespace tmc {
namespace {

constexpr uint32_t BM = 128;
constexpr int kConv = 16, kEpi = 16, kMma = 20, kTok = 21, kWarps = 24;
constexpr uint32_t kMaxTok = 256, kTmemCols = 512, kMaxRing = 8;
constexpr uint32_t kRegion = 224u * 1024u;                       // token slots, then raw slots
constexpr size_t kSmem = kRegion + 1024;
constexpr uint32_t kResident = 96u * 1024u;                      // tokens that the converters round themselves: at most so many bytes of fp16

struct BlockGemm {
    uint32_t M, N, ldc, groups;                                   // groups: K in groups of 256, rounded up
    uint32_t bn, tiles_m, tiles, split;                           // tokens per tile; CTAs that share a tile along K
    uint32_t accs, acc_cols, na, nb, nr;                          // accumulators, their columns; weight and token slots (two stages each), raw slots
    const uint8_t* W;
    const float* A;                                               // resident: the tokens as the caller gave them
    uint32_t row_bytes, K, single, resident;                      // single: no CTA has a second tile
    float* C;
    int* status;
};

struct Bars {
    uint64_t raw_full[kMaxRing], raw_empty[kMaxRing], tok_full[kMaxRing], tok_empty[kMaxRing], a_full[kMaxRing], a_empty[kMaxRing];
    uint64_t acc_full[2], acc_empty[2], tok_ready;
};

// 16 bytes, of which the first `valid` come from memory and the rest are zeros
__device__ __forceinline__ void copy16(uint32_t dst, const uint8_t* src, uint32_t valid) {
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void copies_arrive(uint32_t bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tma_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// K-major rows of 128 bytes, 128-byte swizzle; k = 0..3: the 16 columns of one MMA inside the swizzle atom
__device__ __forceinline__ uint64_t tok_desc(uint32_t saddr, uint32_t k) {
    constexpr uint32_t hi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
    return ((uint64_t)hi << 32) | (uint64_t)((((saddr & 0x3FFFFu) >> 4) | (1u << 16)) + 2u * k);
}
// D[tmem] (+)= A[tmem] B[smem]: 128 rows x bn tokens x 128, the eight MMAs of two stages, issued by the lane with `lead`
// set. The whole warp runs the issuing loop and only the instruction itself is predicated: its operands then stay in
// uniform registers. Inside an `if (lane == 0)` each of them is moved there one by one; a stage took 600 clocks to issue.
__device__ __forceinline__ void mma_pair(uint32_t d, uint32_t a, uint32_t tok, uint32_t tok2, uint32_t idesc, uint32_t acc, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t"
        "setp.ne.b32 p, %18, 0;\n\t"
        "setp.ne.b32 q, %19, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %9, %17, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], %10, %17, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%3], %11, %17, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%4], %12, %17, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%5], %13, %17, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%6], %14, %17, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%7], %15, %17, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%8], %16, %17, t;\n\t}"
        ::"r"(d), "r"(a), "r"(a + 8u), "r"(a + 16u), "r"(a + 24u), "r"(a + 32u), "r"(a + 40u), "r"(a + 48u), "r"(a + 56u),
          "l"(tok_desc(tok, 0)), "l"(tok_desc(tok, 1)), "l"(tok_desc(tok, 2)), "l"(tok_desc(tok, 3)),
          "l"(tok_desc(tok2, 0)), "l"(tok_desc(tok2, 1)), "l"(tok_desc(tok2, 2)), "l"(tok_desc(tok2, 3)),
          "r"(idesc), "r"(acc), "r"(lead) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar, uint32_t lead) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead) : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t t, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]),
        "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
        "r"(v[30]), "r"(v[31]) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t t, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(t));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_cta(uint32_t saddr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_remote4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// A position in a ring of n slots, moved on by one or by `step` (at most n).
struct Pos {
    uint32_t slot = 0, par = 0;
    __device__ __forceinline__ void move(uint32_t step, uint32_t n) { slot += step; if (slot >= n) { slot -= n; par ^= 1u; } }
};

// The part of K that this CTA takes of every tile, in groups.
struct Share {
    uint32_t g0, g1;
    __device__ __forceinline__ Share(const BlockGemm& p, uint32_t rank) { g0 = p.groups * rank / p.split; g1 = p.groups * (rank + 1) / p.split; }
};

// Where a row's group lies in shared memory: its 16-byte lines, from the one it begins in, rows an odd multiple of 16
// bytes apart (the 16-byte reads of 32 rows then meet no bank conflict).
template <int DT, bool AL> struct Raw {
    static constexpr bool kWhole = AL && Codes<DT>::kBytes % 16 == 0;         // groups begin on a line
    static constexpr uint32_t kLines = kWhole ? Codes<DT>::kBytes / 16 : (Codes<DT>::kBytes + 15 + 15) / 16;
    static constexpr uint32_t kPitch = 16 * (kLines | 1u), kSlot = BM * kPitch;
};

// Producers of raw groups, NW warps. A lane keeps to one line and steps through the rows, so that its addresses advance by
// constants: with the line and the row recomputed per copy two warps spent 3000 clocks on a group, all of it latency of the
// index arithmetic.
template <int DT, bool AL, int NW>
__device__ bool request(const BlockGemm& p, Bars* b, uint32_t raw, uint32_t first, uint32_t step, Share sh, uint32_t mine, uint32_t lane, int* gone) {
    using R = Raw<DT, AL>;
    constexpr uint32_t ROWS = 32 * NW / R::kLines, ROUNDS = (BM + ROWS - 1) / ROWS;
    const uint32_t id = mine * 32u + lane, l = id % R::kLines, r0 = id < ROWS * R::kLines ? id / R::kLines : BM;    // BM: nothing to copy
    const uint32_t to = 16u * l, dst0 = raw + r0 * R::kPitch + to;
    const size_t run = (size_t)ROWS * p.row_bytes;
    Pos rp;
    for (uint32_t tile = first; tile < p.tiles; tile += step) {
        const uint32_t n0 = tile / p.tiles_m * BM, rows = min(BM, p.N - n0);
        const uint8_t* begin = p.W + (size_t)(n0 + (r0 < BM ? r0 : 0u)) * p.row_bytes;
        for (uint32_t g = sh.g0; g < sh.g1; ++g) {
            if (!mbar_wait(smem_u32(&b->raw_empty[rp.slot]), rp.par ^ 1u, gone)) return false;
            const uint8_t* at = begin + (size_t)g * Codes<DT>::kBytes;
            uint32_t dst = dst0 + rp.slot * R::kSlot, r = r0;
            const uint32_t left = p.row_bytes - g * Codes<DT>::kBytes;       // bytes from the group's begin to the row's end
            // whole rows and a whole group; lines that reach past it (at most 30 bytes) still lie in the tensor
            if (rows == BM && left >= Codes<DT>::kBytes && (R::kWhole || left >= Codes<DT>::kBytes + 32u || n0 + BM < p.N)) {
                at += to;
#pragma unroll
                for (uint32_t i = 0; i < ROUNDS; ++i) {
                    if (r < BM) copy16(dst, R::kWhole ? at : at - ((uint32_t)(uintptr_t)at & 15u), 16u);
                    at += run; dst += ROWS * R::kPitch; r += ROWS;
                }
            } else {
                for (; r < BM; r += ROWS) {
                    const uint32_t mis = R::kWhole ? 0u : (uint32_t)(uintptr_t)at & 15u;         // the line begins to - mis bytes into the group
                    const uint32_t valid = r < rows && left + mis > to ? min(16u, left + mis - to) : 0u;     // past the end: zeros
                    copy16(dst, valid ? at - mis + to : p.W - ((uintptr_t)p.W & 15u), valid);
                    at += run; dst += ROWS * R::kPitch;
                }
            }
            copies_arrive(smem_u32(&b->raw_full[rp.slot]));
            rp.move(1, p.nr);
        }
    }
    return true;
}

// Eight columns of a token in the order of the weights, columns 8 c .. of stage s of the group at k0. They come from two
// aligned runs of four weights, which lie the same distance apart everywhere.
template <int DT> struct Eight {
    float4 v[2];
    __device__ __forceinline__ void load(const float* a, uint32_t k0, uint32_t s, uint32_t c, uint32_t K) {
        constexpr int at = apart();
        const uint32_t k = k0 + (uint32_t)Codes<DT>::k_of((int)s, (int)(8u * c));
        v[0] = k < K ? __ldg(reinterpret_cast<const float4*>(a + k)) : make_float4(0.f, 0.f, 0.f, 0.f);      // K is a multiple of 32
        v[1] = k + at < K ? __ldg(reinterpret_cast<const float4*>(a + k + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ uint4 rounded() const {
        const float f[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w};
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = as_u32(__floats2half2_rn(f[place(2 * j)], f[place(2 * j + 1)]));
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
private:
    static __host__ __device__ constexpr int apart() { for (int j = 1; j < 8; ++j) if (Codes<DT>::k_of(0, j) >= 4) return Codes<DT>::k_of(0, j) & ~3; return 0; }
    static __host__ __device__ constexpr int place(int j) { return Codes<DT>::k_of(0, j) < 4 ? Codes<DT>::k_of(0, j) : Codes<DT>::k_of(0, j) - apart() + 4; }
};

// The tokens of a tile, this CTA's part of K, rounded into the token slots as a tensor copy would lay them out. Four items
// per thread are requested before the first is used: one at a time cost a DRAM latency each.
template <int DT> __device__ void round_tokens(const BlockGemm& p, uint32_t region, uint32_t m0, Share sh) {
    const uint32_t per = (sh.g1 - sh.g0) * 32u, total = min(p.bn, p.M - m0) * per;
    for (uint32_t base = threadIdx.x; base < total; base += 4u * 32u * kConv) {
        Eight<DT> e[4];
        uint32_t dst[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t i = base + u * 32u * kConv, t = i / per, c = i - t * per;
            if (i < total) e[u].load(p.A + (size_t)(m0 + t) * p.K, (sh.g0 + (c >> 5)) * 256u, (c >> 3) & 3u, c & 7u, p.K);
            dst[u] = region + (c >> 3) * p.bn * 128u + t * 128u + (((c & 7u) ^ (t & 7u)) << 4);
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            if (base + u * 32u * kConv < total) {
                const uint4 w = e[u].rounded();
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst[u]), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
            }
    }
}

// Converters of stage S of every group.
template <int DT, bool AL, int S>
__device__ bool convert(const BlockGemm& p, Bars* b, uint32_t raw, uint32_t tmem, uint32_t first, uint32_t step, Share sh, int q, int lane, int* gone) {
    using R = Raw<DT, AL>;
    bool ok = true;
    Pos rp, ap;
    ap.move(S >> 1, p.na);
    const uint32_t lanes = (uint32_t)q * 32u, row = raw + (lanes + lane) * R::kPitch;
    for (uint32_t tile = first; tile < p.tiles; tile += step)
        for (uint32_t g = sh.g0; g < sh.g1; ++g) {
            uint32_t o[32];
            if (!mbar_wait(smem_u32(&b->raw_full[rp.slot]), rp.par, gone)) ok = false;
            uint32_t off = 0;
            if constexpr (!R::kWhole) {
                const uint32_t r = tile / p.tiles_m * BM + lanes + lane;
                off = ((uint32_t)(uintptr_t)p.W + r * p.row_bytes + g * Codes<DT>::kBytes) & 15u;
            }
            Codes<DT>::template stage<S, AL>(row + rp.slot * R::kSlot, off, o);
            __syncwarp();
            mbar_arrive_if(smem_u32(&b->raw_empty[rp.slot]), lane == 0);
            if (!mbar_wait(smem_u32(&b->a_empty[ap.slot]), ap.par ^ 1u, gone)) ok = false;
            fence_after();
            tmem_st32(tmem + (lanes << 16) + kTmemCols - 64u * (ap.slot + 1) + 32u * (S & 1), o);
            fence_before();
            __syncwarp();
            mbar_arrive_if(smem_u32(&b->a_full[ap.slot]), lane == 0);
            rp.move(1, p.nr);
            ap.move(2, p.na);
        }
    return ok;
}

template <int DT, bool AL>
__global__ void __launch_bounds__(32 * kWarps, 1)
gemm_blocks(const __grid_constant__ CUtensorMap tm_tok, const BlockGemm p) {
    extern __shared__ uint8_t smem_dyn[];
    __shared__ __align__(8) Bars bars;
    __shared__ uint32_t tmem_slot;
    __shared__ int gone;
    const uint32_t region = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: known to be uniform
    const uint32_t tok_bytes = p.bn * 256u, raw = region + p.nb * tok_bytes;
    if (threadIdx.x == 0) {
        gone = 0;
        for (uint32_t i = 0; i < kMaxRing; ++i) {
            mbar_init(smem_u32(&bars.raw_full[i]), p.single ? 192 : 64); mbar_init(smem_u32(&bars.raw_empty[i]), kConv);
            mbar_init(smem_u32(&bars.tok_full[i]), 1); mbar_init(smem_u32(&bars.tok_empty[i]), 1);
            mbar_init(smem_u32(&bars.a_full[i]), 8); mbar_init(smem_u32(&bars.a_empty[i]), 1);
        }
        mbar_init(smem_u32(&bars.tok_ready), kConv);
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&bars.acc_full[i]), 1); mbar_init(smem_u32(&bars.acc_empty[i]), 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t rank = p.split > 1 ? cluster_rank() : 0u;
    const uint32_t first = blockIdx.x / p.split, step = gridDim.x / p.split;
    const Share sh(p, rank);
    bool ok = true;

    if (warp < kConv) {
        if (p.resident) {
            round_tokens<DT>(p, region, first % p.tiles_m * p.bn, sh);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            mbar_arrive_if(smem_u32(&bars.tok_ready), lane == 0);
        }
        switch (warp >> 2) {
            case 0: ok = convert<DT, AL, 0>(p, &bars, raw, tmem, first, step, sh, warp & 3, lane, &gone); break;
            case 1: ok = convert<DT, AL, 1>(p, &bars, raw, tmem, first, step, sh, warp & 3, lane, &gone); break;
            case 2: ok = convert<DT, AL, 2>(p, &bars, raw, tmem, first, step, sh, warp & 3, lane, &gone); break;
            default: ok = convert<DT, AL, 3>(p, &bars, raw, tmem, first, step, sh, warp & 3, lane, &gone); break;
        }
    } else if (warp > kTok) {
        const uint32_t mine = (uint32_t)(warp - kTok - 1);
        ok = p.single ? request<DT, AL, 6>(p, &bars, raw, first, step, sh, mine, (uint32_t)lane, &gone)
                      : request<DT, AL, 2>(p, &bars, raw, first, step, sh, mine, (uint32_t)lane, &gone);
    } else if (warp == kTok) {
        if (lane == 0 && !p.resident) {
            asm volatile("griddepcontrol.wait;" ::: "memory");   // the launch before this one writes the fp16 tokens
            Pos tp;
            for (uint32_t tile = first; tile < p.tiles && ok; tile += step)
                for (uint32_t h = 0; h < 2 * (sh.g1 - sh.g0); ++h) {
                    if (!mbar_wait(smem_u32(&bars.tok_empty[tp.slot]), tp.par ^ 1u, &gone)) { ok = false; break; }
                    const uint32_t bar = smem_u32(&bars.tok_full[tp.slot]);
                    mbar_expect_tx(bar, tok_bytes);
                    tma_3d(region + tp.slot * tok_bytes, &tm_tok, 0, (int)(tile % p.tiles_m * p.bn), (int)(4 * sh.g0 + 2 * h), bar);
                    tp.move(1, p.nb);
                }
        }
    } else if (warp == kMma) {
        const uint32_t idesc = (1u << 4) | ((p.bn >> 3) << 17) | ((BM >> 4) << 24);      // fp16 x fp16 -> fp32, K-major
        const uint32_t lead = elect_one(), pairs = 2 * (sh.g1 - sh.g0);
        Pos ap, tp;
        uint32_t count = 0;
        bool ta = false, tt = false;                             // what the probes issued with the previous pair said
        if (p.resident && !mbar_wait(smem_u32(&bars.tok_ready), 0, &gone)) ok = false;
        for (uint32_t tile = first; tile < p.tiles && ok; tile += step, ++count) {
            const uint32_t acc = p.accs == 2 ? count & 1u : 0u, use = p.accs == 2 ? count >> 1 : count;
            if (!mbar_wait(smem_u32(&bars.acc_empty[acc]), (use & 1u) ^ 1u, &gone)) { ok = false; break; }
            const uint32_t d = tmem + acc * p.acc_cols;
            for (uint32_t h = 0; h < pairs; ++h) {
                if (!p.resident && !tt && !mbar_wait(smem_u32(&bars.tok_full[tp.slot]), tp.par, &gone)) { ok = false; break; }
                if (!ta && !mbar_wait(smem_u32(&bars.a_full[ap.slot]), ap.par, &gone)) { ok = false; break; }
                fence_after();
                const Pos a0 = ap, t0 = tp;
                ap.move(1, p.na);
                tp.move(1, p.nb);
                if (!p.resident) tt = mbar_test(smem_u32(&bars.tok_full[tp.slot]), tp.par);
                ta = mbar_test(smem_u32(&bars.a_full[ap.slot]), ap.par);
                const uint32_t t = region + t0.slot * tok_bytes;
                mma_pair(d, tmem + kTmemCols - 64u * (a0.slot + 1), t, t + p.bn * 128u, idesc, h, lead);
                mma_commit(smem_u32(&bars.a_empty[a0.slot]), lead);
                if (!p.resident) mma_commit(smem_u32(&bars.tok_empty[t0.slot]), lead);
            }
            mma_commit(smem_u32(&bars.acc_full[acc]), lead);
        }
    } else if (p.single && !request<DT, AL, 6>(p, &bars, raw, first, step, sh, (uint32_t)(warp - kEpi + 2), (uint32_t)lane, &gone)) {
        ok = false;
    }
    if (warp >= kEpi && warp < kMma && p.split == 1) {
        const uint32_t q = (uint32_t)warp & 3u;
        if (!p.resident) asm volatile("griddepcontrol.wait;" ::: "memory");       // C may still be read by what ran before that launch
        uint32_t count = 0;
        for (uint32_t tile = first; tile < p.tiles; tile += step, ++count) {
            const uint32_t acc = p.accs == 2 ? count & 1u : 0u, use = p.accs == 2 ? count >> 1 : count;
            if (!mbar_wait(smem_u32(&bars.acc_full[acc]), use & 1u, &gone)) { ok = false; break; }
            fence_after();
            const uint32_t n = tile / p.tiles_m * BM + q * 32u + lane, m0 = tile % p.tiles_m * p.bn;
            for (uint32_t c0 = 0; c0 < p.bn && m0 + c0 < p.M; c0 += 16) {
                uint32_t v[16];
                tmem_ld16(tmem + acc * p.acc_cols + c0 + (q << 21), v);
                float* out = p.C + (size_t)(m0 + c0) * p.ldc + n;
                if (n < p.N) {
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j)
                        if (m0 + c0 + j < p.M) out[(size_t)j * p.ldc] = __uint_as_float(v[j]);
                }
            }
            fence_before();
            __syncwarp();
            mbar_arrive_if(smem_u32(&bars.acc_empty[acc]), lane == 0);
        }
    }
    if (p.split > 1) {
        // One tile per cluster. Its tokens are dealt out to the CTAs: each collects all partial sums of its own, in the
        // memory that the rings no longer need, and adds them in the order of K.
        const uint32_t tile = first, n0 = tile / p.tiles_m * BM, m0 = tile % p.tiles_m * p.bn;
        const uint32_t mine = ((p.bn + p.split - 1) / p.split + 3) & ~3u, pitch = 4u * (mine + 4u);     // tokens per CTA; bytes from row to row
        const uint32_t q = (uint32_t)warp & 3u, live = min(p.bn, p.M - m0);
        const bool epi = warp >= kEpi && warp < kMma;
        if (epi) {
            if (!mbar_wait(smem_u32(&bars.acc_full[0]), 0, &gone)) ok = false;
            fence_after();
        }
        cluster_sync();                                          // every CTA of the tile is through with its rings
        if (epi) {
            uint32_t owner = 0, t = 0;                           // whose part the column belongs to, its place there
            uint32_t to = map_cta(region + (rank * BM + q * 32u + lane) * pitch, 0);
            for (uint32_t c0 = 0; c0 < live; c0 += 16) {
                uint32_t v[16];
                tmem_ld16(tmem + c0 + (q << 21), v);
#pragma unroll
                for (uint32_t j = 0; j < 16; j += 4) {
                    if (c0 + j < live) st_remote4(to + 4u * t, v[j], v[j + 1], v[j + 2], v[j + 3]);
                    t += 4;
                    if (t == mine) { t = 0; ++owner; to = map_cta(region + (rank * BM + q * 32u + lane) * pitch, owner < p.split ? owner : 0u); }
                }
            }
        }
        cluster_sync();
        if (!p.resident) asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t t0 = rank * mine;
        for (uint32_t i = threadIdx.x; i < mine / 4 * BM; i += 32 * kWarps) {
            const uint32_t t = i / BM * 4, r = i % BM, m = m0 + t0 + t;
            if (t0 + t >= live || n0 + r >= p.N) continue;
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t c = 0; c < p.split; ++c) {
                const uint4 x = lds_line(region + (c * BM + r) * pitch + 4u * t);
                s.x += __uint_as_float(x.x); s.y += __uint_as_float(x.y); s.z += __uint_as_float(x.z); s.w += __uint_as_float(x.w);
            }
            float* out = p.C + (size_t)m * p.ldc + n0 + r;
            out[0] = s.x;
            if (t0 + t + 1 < live) out[p.ldc] = s.y;
            if (t0 + t + 2 < live) out[2 * (size_t)p.ldc] = s.z;
            if (t0 + t + 3 < live) out[3 * (size_t)p.ldc] = s.w;
        }
    }
    if (!ok) *(volatile int*)p.status = 2;
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_before();
    __syncthreads();
    if (gone && threadIdx.x == 0) {                              // a wait ran out: copies may be in flight, a last bounded chance to land
        gone = 0;
        for (uint32_t i = 0; i < kMaxRing; ++i)
            for (uint32_t par = 0; par < 2; ++par) (void)mbar_wait(smem_u32(&bars.tok_full[i]), par, &gone, 20000000ull);
    }
    if (warp == kMma) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// Tokens as the weights' order wants them: [M][Kp] fp16, every 64 columns permuted by k_of, K rounded up to 64 with zeros.
template <int DT>
__global__ void __launch_bounds__(256) gemm_tokens(const float* __restrict__ A, __half* __restrict__ Ah, uint32_t K, uint32_t Kp, uint32_t total) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;          // eight columns of one token
    if (i >= total) return;
    const uint32_t per = Kp / 8, m = i / per, c = i - m * per;
    Eight<DT> e;
    e.load(A + (size_t)m * K, (c >> 5) * 256u, (c >> 3) & 3u, c & 7u, K);
    reinterpret_cast<uint4*>(Ah)[i] = e.rounded();
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode() {
    static const EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? (EncodeFn)p : nullptr;
    }();
    return fn;
}

// Token tile and split of K. A tile's time is modelled per stage of 64 columns: the converters need about kStageClocks
// (one figure between the formats: 160-190 for Q4_0, about 500 for Q6_K),
// the tensor pipe two clocks per token column; emptying an accumulator costs about 1000 + 10 per column and overlaps the
// next tile only when two fit beside the weight stages (up to 192 tokens).
void plan(BlockGemm& p, uint32_t raw_bytes, uint32_t sms) {
    constexpr uint32_t kStageClocks = 280;
    const uint32_t rt = (p.N + BM - 1) / BM;
    unsigned long long best = ~0ull;
    for (uint32_t bn = kMaxTok; bn >= 16; bn -= 16) {
        if (bn - 16 >= p.M || (bn < 64 && p.M > 64)) continue;
        const uint32_t tm = (p.M + bn - 1) / bn, tiles = rt * tm;
        uint32_t split = sms / tiles ? sms / tiles : 1u;
        if (split > 8) split = 8;
        if (split > p.groups) split = p.groups;
        const uint32_t waves = (tiles * split + sms - 1) / sms, cols = (bn + 31) / 32 * 32, accs = waves > 1 && 2 * cols + 128 <= kTmemCols ? 2 : 1;
        const uint32_t stage = 2 * bn > kStageClocks ? 2 * bn : kStageClocks, empty = 1000 + 10 * bn;
        const unsigned long long main = 4ull * stage * ((p.groups + split - 1) / split);
        const unsigned long long cost = waves * main + (accs == 2 ? empty : (unsigned long long)waves * empty);
        if (cost < best) { best = cost; p.bn = bn; p.tiles_m = tm; p.tiles = tiles; p.split = split; p.accs = accs; p.acc_cols = cols; }
    }
    p.na = (kTmemCols - p.accs * p.acc_cols) / 64;
    if (p.na > 4) p.na = 4;
    const uint32_t tok = p.bn * 256, pairs = 2 * ((p.groups + p.split - 1) / p.split);
    p.single = p.split > 1 || p.tiles <= sms;
    p.nb = (kRegion - 2 * raw_bytes) / tok;
    if (p.nb > 6) p.nb = 6;
    p.resident = p.single && (uint64_t)pairs * tok <= kResident;
    if (p.resident) p.nb = pairs;
    p.nr = (kRegion - p.nb * tok) / raw_bytes;
    if (p.nr > kMaxRing) p.nr = kMaxRing;
}

template <int DT, bool AL>
bool launch_rows(BlockGemm p, const float* A, uint32_t K, __half* Ah, cudaStream_t st) {
    const EncodeFn fn = encode();
    if (!fn) return fail("gemm: cuTensorMapEncodeTiled is unavailable");
    plan(p, Raw<DT, AL>::kSlot, (uint32_t)device_sm_count());
    CUtensorMap tok = {};
    const uint32_t Kp = (K + 63) / 64 * 64;
    if (!p.resident) {
        const cuuint64_t dims[3] = {64, p.M, Kp / 64}, strides[2] = {(cuuint64_t)Kp * 2, 128};
        const cuuint32_t ones[3] = {1, 1, 1}, box[3] = {64, p.bn, 2};
        const CUresult r = fn(&tok, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, Ah, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail("gemm: tensor map encode failed (%d)", (int)r);
    }
    static const cudaError_t attr = cudaFuncSetAttribute(gemm_blocks<DT, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (attr != cudaSuccess) return fail("gemm: shared memory attribute: %s", cudaGetErrorString(attr));
    if (!p.resident) {
        const uint32_t total = (uint32_t)((uint64_t)p.M * Kp / 8);
        gemm_tokens<DT><<<(total + 255) / 256, 256, 0, st>>>(A, Ah, K, Kp, total);
        note_launch();
        if (!check_launch("gemm_tokens")) return false;
    }
    const uint32_t sms = (uint32_t)device_sm_count();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.split > 1 ? p.tiles * p.split : p.tiles < sms ? p.tiles : sms);
    cfg.blockDim = dim3(32 * kWarps); cfg.dynamicSmemBytes = kSmem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    if (p.split > 1) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = p.split; at[cfg.numAttrs].val.clusterDim.y = 1; at[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    if (!p.resident) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        ++cfg.numAttrs;
    }
    cfg.attrs = at;
    if (cudaLaunchKernelEx(&cfg, gemm_blocks<DT, AL>, tok, p) != cudaSuccess) return check_launch("gemm_blocks");
    note_launch();
    return check_launch("gemm_blocks");
}
template <int DT> bool launch_dt(const BlockGemm& p, const float* A, uint32_t K, __half* Ah, cudaStream_t st) {
    if ((uintptr_t)p.W % 16 == 0 && p.row_bytes % 16 == 0) return launch_rows<DT, true>(p, A, K, Ah, st);
    if constexpr (DT == 5 || DT == 8) return fail("gemm: Q4_K and Q5_K rows start on 16-byte boundaries here");
    else return launch_rows<DT, false>(p, A, K, Ah, st);
}

}  // namespace

bool gemm_blocks_takes(const uint8_t* W, unsigned M, unsigned N, unsigned K, unsigned dtype, size_t scratch_bytes) {
    const uint64_t tok = (uint64_t)M * ((K + 63) / 64 * 64);
    if (tok * 2 > scratch_bytes || tok / 8 > 0xffffff00ull || (uint64_t)N + 128 > 0xffffffffull) return false;
    if (dtype == DT_Q5_K || dtype == DT_Q4_K) return (uintptr_t)W % 16 == 0;       // their rows are whole 16-byte lines
    return dtype == DT_Q8_0 || dtype == DT_Q4_0 || dtype == DT_Q4_1 || dtype == DT_Q6_K || dtype == DT_GGUF_Q4_0;
}

bool launch_gemm_blocks(const float* A, const uint8_t* W, float* C, unsigned ldc, unsigned M, unsigned N, unsigned K, unsigned dtype,
                        void* Ah, cudaStream_t st) {
    BlockGemm p = {};
    p.M = M; p.N = N; p.ldc = ldc; p.groups = (K + 255) / 256; p.C = C; p.status = device_status_word();
    p.W = W; p.A = A; p.K = K; p.row_bytes = K / block_elems(dtype) * block_bytes(dtype);
    __half* h = (__half*)Ah;
    switch (dtype) {
        case DT_Q8_0: return launch_dt<0>(p, A, K, h, st);
        case DT_Q4_0: return launch_dt<1>(p, A, K, h, st);
        case DT_Q4_1: return launch_dt<4>(p, A, K, h, st);
        case DT_Q5_K: return launch_dt<5>(p, A, K, h, st);
        case DT_Q4_K: return launch_dt<8>(p, A, K, h, st);
        case DT_GGUF_Q4_0: return launch_dt<9>(p, A, K, h, st);
        default: return launch_dt<6>(p, A, K, h, st);
    }
}

}  // namespace tmc
