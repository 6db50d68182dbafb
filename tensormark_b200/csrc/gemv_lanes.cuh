// gemv_lanes.cuh — how a warp turns a tile of block-quantized rows into dot products on the integer tensor cores.
//
// Unit of work: 16 weight rows x one "group" of 256 weights, one m16n8k32 int8 MMA sequence of a warp. In that MMA's
// fragment layout thread (g, t) = (lane / 4, lane % 4) supplies, for every k-step, eight bytes of row g and eight of
// row g + 8, and receives columns 2t and 2t + 1 of both rows. Which weights the k index names is free, so thread t is
// given the quarter t of the group (64 weights) of its two rows, exactly the bytes it has loaded, and the activations
// are laid out block-diagonally: column 2t + p holds plane p of quarter t under the k indices that thread t supplies
// and zero everywhere else. Column 2t + p of the product is then the dot product of quarter t alone, and it arrives
// in the thread that holds the block scales of that quarter: no cross-lane traffic until a row is finished. Three
// quarters of the multiplications are by zero and that costs nothing: measured, one MMA per 1.07 ns and SM, 512
// weights each, is 40 TB/s of 4-bit blocks against 6.5 TB/s of HBM. What counts is instructions per weight: the
// dp4a lanes this replaces issued 160 per 2048 weights of one row, these about 55 (Q4_0).
//
// Arithmetic. The integer codes of a block are never converted one by one. The activations of every 32-block are
// re-expressed once per kernel as block floating point: a scale s = max|x|/127 and kPlanes signed 8-bit planes with
//     x[i] ~= s * (a1[i] + a2[i]/128),
// error <= 2^-15 * max|x| per activation (3.1e-5 of the block maximum, which for activations of one scale is below
// 1e-4 * sum|w x| even if every rounding error lined up with the sign of its weight, an order inside the 1e-3
// contract; measured ~2e-6). A block's dot product is two exact integer dot products, 128 S1 + S2 in one integer, one
// conversion to fp32, times the block scales, added to the row's fp32 accumulator: exact within a block, fp32 across
// blocks, like the reference's per-block partial sums (tensormark/llama.h:1877-1895). Zero points (Q4_0, Q6_K) and mins
// (Q4_1, Q4_K, Q5_K) multiply the true fp32 sums of x, so nothing depends on the planes' rounding beyond that bound. NaN or infinite activations poison the block scale and
// therefore the output, as a floating-point chain would.
//
// Everything here but the MMA itself is __host__ __device__: the test-suite replays the maps on a CPU against the
// checker before a GPU ever runs them.
//
// Layouts decoded are the serialized blocks of tensormark/quant.h:35-49 and 214-245; the GPU kernels replaced are the
// cooperative-row GEMVs of tensormark/metal.h:359-440 (Q4_0), 641-679 (Q4_1), 708-754 (Q5_K), 775-822 (Q6_K).
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#include <cuda_fp16.h>
#define TM_HD __host__ __device__ __forceinline__
#else
#include <math.h>
#define TM_HD inline
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct uint2 { unsigned x, y; };
struct uint4 { unsigned x, y, z, w; };
#endif

namespace tmc {

constexpr int kPlanes = 2;                                  // int8 planes of the activations: columns 2t and 2t + 1 of the MMA

// ---- primitives with host emulation ----------------------------------------
TM_HD float as_float(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f; memcpy(&f, &u, 4); return f;
#endif
}
TM_HD uint32_t as_uint(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u; memcpy(&u, &f, 4); return u;
#endif
}
TM_HD float fma1(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}
TM_HD float half_to_float(uint32_t h) {
#if defined(__CUDA_ARCH__)
    return __half2float(__ushort_as_half((unsigned short)h));
#else
    const uint32_t s = (h & 0x8000u) << 16, e = (h >> 10) & 31u, m = h & 1023u;
    if (e == 31u) return as_float(s | 0x7f800000u | (m << 13));
    if (e != 0u) return as_float(s | ((e + 112u) << 23) | (m << 13));
    const float mag = (float)m * 0x1p-24f;
    return as_float(s | as_uint(mag));
#endif
}
TM_HD uint32_t funnel_r(uint32_t lo, uint32_t hi, uint32_t sh) {   // sh < 32
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, sh);
#else
    return sh ? ((lo >> sh) | (hi << (32 - sh))) : lo;
#endif
}
#if !defined(__CUDACC__)
// c + sum of four (signed / unsigned byte of a) * (signed byte of b)
inline int dp4a_ss(uint32_t a, uint32_t b, int c) {
    for (int k = 0; k < 4; ++k) c += (int)(int8_t)((a >> (8 * k)) & 0xff) * (int)(int8_t)((b >> (8 * k)) & 0xff);
    return c;
}
inline int dp4a_us(uint32_t a, uint32_t b, int c) {
    for (int k = 0; k < 4; ++k) c += (int)((a >> (8 * k)) & 0xff) * (int)(int8_t)((b >> (8 * k)) & 0xff);
    return c;
}
#endif
// ---- block floating point of 32 activations ----------------------------------
// Block scale from the block's max |x| (and whether the block holds NaN/inf): x ~= s * (a[0] + a[1]/128). A poisoned
// block gets s = NaN so every output that touches it is NaN; a block of zeros (or of values too small to scale) gets
// s = 0.
TM_HD float block_scale(float amax, bool bad, float& inv) {
    if (bad) { inv = 0.f; return as_float(0x7fc00000u); }
    if (!(amax >= 1.0e-30f)) { inv = 0.f; return 0.f; }
    inv = 127.0f / amax;
    return amax * (1.0f / 127.0f);                          // s * inv == 1 to within 2^-23, far below the plane truncation
}
// The two signed bytes of one activation under its block's inverse scale: the activation is rounded once to a multiple
// of s / 128 (X = round(v / s * 128)) and X is split into signed digits base 128, X = a1 * 128 + a2, a1 in [-127, 127],
// a2 in [-64, 64]. Integer arithmetic after one rounding, which on the GPU is the add of 1.5 * 2^23 (the integer lands
// in the low mantissa bits).
TM_HD void quantize_elem(float v, float inv, int8_t* a) {
    float r = inv == 0.f ? 0.f : v * inv;                   // inv is 0 for empty and for poisoned blocks
    r = r > 127.f ? 127.f : (r < -127.f ? -127.f : r);
#if defined(__CUDA_ARCH__)
    const int X = __float_as_int(__fadd_rn(r * 128.0f, 12582912.0f)) - 0x4B400000;
#else
    const int X = (int)lrintf(r * 128.0f);
#endif
    const int a1 = (X + 64) >> 7;
    a[0] = (int8_t)a1; a[1] = (int8_t)(X - a1 * 128);
}

// quantize_elem of four neighbours, packed: first planes in q1, second in q2, low byte first. The sums v * inv * 128 + 64
// land in the low mantissa bits as Y = 128 a1 + (a2 + 64); two of them share a register, a1 being bits 7..14 and a2 + 64
// bits 0..6 of each half. No clamp: |v| * inv is 127 to within rounding. (A poisoned block has inv = 0, so a NaN may
// leave any bytes; its scale is NaN.)
#if defined(__CUDACC__)
__device__ __forceinline__ void quantize_quad(float x, float y, float z, float w, float inv, uint32_t& q1, uint32_t& q2) {
    const float s = inv * 128.0f, magic = 12582912.0f + 64.0f;
    const uint32_t y0 = __float_as_uint(__fadd_rn(__fmul_rn(x, s), magic)), y1 = __float_as_uint(__fadd_rn(__fmul_rn(y, s), magic));
    const uint32_t y2 = __float_as_uint(__fadd_rn(__fmul_rn(z, s), magic)), y3 = __float_as_uint(__fadd_rn(__fmul_rn(w, s), magic));
    const uint32_t p01 = __byte_perm(y0, y1, 0x5410), p23 = __byte_perm(y2, y3, 0x5410);
    q1 = __byte_perm(p01 >> 7, p23 >> 7, 0x6420);
    const uint32_t f = (__byte_perm(p01, p23, 0x6420) & 0x7F7F7F7Fu) ^ 0x40404040u;      // a2 in seven bits, two's complement
    q2 = f | ((f & 0x40404040u) << 1);
}
// Two more planes: what rounding to multiples of s / 128 left, in multiples of s / 2^21: x ~= s (a1 + a2/128 + a3/2^14 +
// a4/2^21), as close as fp32 holds x.
__device__ __forceinline__ void quantize_rest(float x, float y, float z, float w, float inv, uint32_t& q3, uint32_t& q4) {
    const float s = inv * 128.0f, magic = 12582912.0f;
    auto rest = [&](float v) { const float t = __fmul_rn(v, s); return __fmul_rn(__fadd_rn(t, -__fadd_rn(__fadd_rn(t, magic), -magic)), 128.0f); };   // exact, |rest| <= 64
    quantize_quad(rest(x), rest(y), rest(z), rest(w), 1.0f, q3, q4);
}
#endif

// Loads of weight bytes. On the GPU the bytes lie in shared memory and an address is the 32-bit one (SPtr): generic
// pointers cost the row loop a handful of instructions per use. On the host it is a pointer.
#if defined(__CUDACC__)
using SPtr = uint32_t;
__device__ __forceinline__ uint32_t ld4(SPtr p) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p)); return v; }
__device__ __forceinline__ uint2 ld8(SPtr p) { uint2 v; asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(p)); return v; }
__device__ __forceinline__ uint4 ld16(SPtr p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld2(SPtr p) { uint16_t v; asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p)); return v; }
#define TM_SD __device__ __forceinline__
#else
using SPtr = const uint8_t*;
inline uint32_t ld4(SPtr p) { uint32_t v; memcpy(&v, p, 4); return v; }
inline uint2 ld8(SPtr p) { uint2 v; memcpy(&v, p, 8); return v; }
inline uint4 ld16(SPtr p) { uint4 v; memcpy(&v, p, 16); return v; }
inline uint32_t ld2(SPtr p) { uint16_t v; memcpy(&v, p, 2); return v; }
#define TM_SD inline
#endif
// NW words from an even address; AL: the address is known to be a multiple of 4.
template <int NW, bool AL> TM_SD void load_words(SPtr p, uint32_t (&w)[NW]) {
#if defined(__CUDACC__)
    if constexpr (!AL) {
        const uint32_t mis = p & 2u, sh = mis * 8u, q = p - mis;
        uint32_t lo = ld4(q);
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            const uint32_t hi = (i + 1 < NW || mis) ? ld4(q + 4 * (i + 1)) : 0u;
            w[i] = funnel_r(lo, hi, sh);
            lo = hi;
        }
        return;
    }
#endif
#pragma unroll
    for (int i = 0; i < NW; ++i) w[i] = ld4(p + 4 * i);
}
TM_SD uint32_t odd_half(SPtr p) {                          // 2 when p is even but no multiple of 4 (the host reads any address)
#if defined(__CUDACC__)
    return p & 2u;
#else
    (void)p;
    return 0u;
#endif
}
TM_HD uint32_t join16(uint32_t lo, uint32_t hi) {           // upper half of lo | lower half of hi << 16
#if defined(__CUDA_ARCH__)
    return __byte_perm(lo, hi, 0x5432);
#else
    return (lo >> 16) | (hi << 16);
#endif
}

// ---- x image -----------------------------------------------------------------------------------------------------
// Per group of 256 activations kXGroupWords words: 128 words of plane bytes, then eight floats per quarter t. MMA m
// (0..7) of the sequence multiplies the code words 2m and 2m + 1 of every quarter; its two words for (quarter t, plane
// p) lie at word 32 (m / 2) + 4 (2t + p) + 2 (m % 2), so the eight threads of a warp that hold non-zero columns fetch
// the operands of two MMAs with one conflict-free 16-byte load. The floats are what the format's combine() wants:
// {scale, scale, sum term, sum term} of the quarter's two 32-blocks; for Q6_K the scales of its four runs and their four
// sum terms.
constexpr int kXGroupWords = 160;
constexpr int kGroupW = 256;                                // weights per group

// word of the image that holds code word c (0..15) of quarter t, plane p
TM_HD uint32_t x_word(uint32_t group, uint32_t t, uint32_t c, uint32_t p) {
    const uint32_t m = c >> 1;
    return group * (uint32_t)kXGroupWords + 32u * (m >> 1) + 4u * (2u * t + p) + 2u * (m & 1u) + (c & 1u);
}

// A format's Lane. The row loop runs out of ALU slots (LOP3, SHF and PRMT issue at half rate) before anything else, so
// codes are masked out of the bytes where they lie and shifted afterwards, once per integer sum: the parts of a code -
// low nibbles, high nibbles, high bits - go through MMAs of their own and merge() adds their sums, scaled.
//   GB            bytes of a group;  NR  results per quarter (32-blocks, or runs with a scale of their own)
//   NACC, MPA     integer sums per quarter and MMAs per sum; SIGNED  code bytes are signed
//   code_pos      (x word, byte) under which element e of the group is multiplied, e's quarter
//   load          one row's quarter t: its raw words and its scales
//   code          code word i of sum k; xw(k): the x word that its first one meets
//   merge         the sums (128 S1 + S2 each) into results
//   combine       row accumulator + the quarter's contribution from the results and the eight floats
// STEP_*, UNIT_W, LANE_* describe the same thing as a step of eight groups over 32 lanes (lane = 4 group + t).
template <int DT> struct Lane;
#if defined(__CUDACC__)
#define TM_LANE_HOST(DT)
#else
template <int DT> struct LaneHost { static float dot(const uint8_t* quarter, const uint32_t* w, int t, int nvalid); };
// lane's share of a step for the host replay: p = the lane's own bytes (two 32-blocks) or the step's first super-block
#define TM_LANE_HOST(DT)                                                                                    \
    static float dot(const uint8_t* p, const X& x, int lane, int nvalid) {                                  \
        if (LANE_UNITS == 2) return LaneHost<DT>::dot(p, x.w, lane & 3, nvalid);                            \
        return (lane >> 2) < nvalid ? LaneHost<DT>::dot(p + (lane >> 2) * GB, x.w, lane & 3, 2) : 0.f;      \
    }
#endif

// What the 32-weight formats and the 32-weight sub-blocks of Q4_K / Q5_K share: quarter t = 32-blocks 2t, 2t + 1.
template <int GROUP_BYTES, bool SUMS> struct LanePairs {
    static constexpr int GB = GROUP_BYTES, NR = 2;
    static constexpr bool SIGNED = false;
    static constexpr int STEP_W = 2048, STEP_BYTES = 8 * GROUP_BYTES, XW = kXGroupWords / 4;
    static constexpr bool NEEDS_SUMS = SUMS;
    struct X { uint32_t w[XW]; };
    static TM_HD void mask_d(float (&d)[2], int nvalid) { if (nvalid < 1) d[0] = 0.f; if (nvalid < 2) d[1] = 0.f; }
    static TM_HD void put_scalars(uint32_t* units, uint32_t b, float s, float s32) {
        uint32_t* f = units + (b >> 3) * (uint32_t)kXGroupWords + 128u + 8u * ((b & 7u) >> 1) + (b & 1u);
        f[0] = as_uint(s);
        f[2] = SUMS ? as_uint(s32) : 0u;
    }
};
template <typename L> TM_HD uint32_t plane_byte_of(uint32_t e, int p) {          // byte offset of plane p of element e
    uint32_t t, c, byte;
    L::code_pos(e & 255u, t, c, byte);
    return 4u * x_word(e >> 8, t, c, (uint32_t)p) + byte;
}

// ---- Q8_0: 34-byte blocks [d:2][q:32], w = q * d ------------------------------------------------------------------
template <> struct Lane<0> : LanePairs<272, false> {
    static constexpr int UNIT_W = 32, LANE_UNITS = 2, LANE_BYTES = 68;
    static constexpr int NRAW = 17, NACC = 2, MPA = 4;
    static constexpr bool SIGNED = true;
    struct Meta { float d[2]; };
    static TM_HD void code_pos(uint32_t e, uint32_t& t, uint32_t& c, uint32_t& byte) { t = e >> 6; c = (e & 63u) >> 2; byte = e & 3u; }
    static TM_HD uint32_t plane_byte(uint32_t e, int p) { return plane_byte_of<Lane<0>>(e, p); }
    static TM_HD void store_quad(uint32_t* units, uint32_t e0, int p, uint32_t packed) { units[plane_byte(e0, p) >> 2] = packed; }
    static TM_HD void scalars(uint32_t* units, uint32_t b, int lane, int, float s, float, float, float s32) {
        if (lane == 0) put_scalars(units, b, s * (1.0f / 128.0f), s32);
    }
    template <bool AL> static TM_SD void load(SPtr p, int, uint32_t (&w)[17], Meta& m) {
        load_words<17, AL>(p, w);
        m.d[0] = half_to_float(w[0] & 0xffffu); m.d[1] = half_to_float(w[8] >> 16);
    }
    static TM_HD uint32_t code(const uint32_t (&w)[17], int k, int i, int) { return k == 0 ? join16(w[i], w[i + 1]) : w[9 + i]; }
    static constexpr TM_HD int xw(int k) { return 8 * k; }
    static TM_HD void merge(const int (&c)[2], int, int (&S)[2]) { S[0] = c[0]; S[1] = c[1]; }
    static TM_HD void mask(Meta& m, int nvalid) { mask_d(m.d, nvalid); }
    static TM_HD float combine(const float (&S)[2], const Meta& m, const float4 xs, const float4, float acc) {
        return fma1(m.d[1], xs.y * S[1], fma1(m.d[0], xs.x * S[0], acc));
    }
    TM_LANE_HOST(0)
};

// ---- Q4_0: 18-byte blocks [d:2][qs:16], byte j = elements 2j (low) | 2j+1 (high), w = (n-8)*d. Sums per block: the low
// nibbles, and 16 times the high ones; the result is 16 times the block's. The sum term is -8 sum(x).
template <> struct Lane<1> : LanePairs<144, true> {
    static constexpr int UNIT_W = 32, LANE_UNITS = 2, LANE_BYTES = 36;
    static constexpr int NRAW = 9, NACC = 4, MPA = 2;
    struct Meta { float d[2]; };
    static TM_HD void code_pos(uint32_t e, uint32_t& t, uint32_t& c, uint32_t& byte) {
        const uint32_t j = e & 31u;
        t = e >> 6; c = 8u * ((e >> 5) & 1u) + 4u * (j & 1u) + (j >> 3); byte = (j >> 1) & 3u;
    }
    static TM_HD uint32_t plane_byte(uint32_t e, int p) { return plane_byte_of<Lane<1>>(e, p); }
    static TM_HD void store_quad(uint32_t* units, uint32_t e0, int p, uint32_t packed) {      // elements e0, e0+2 | e0+1, e0+3
        uint8_t* q = reinterpret_cast<uint8_t*>(units);
        *reinterpret_cast<uint16_t*>(q + plane_byte(e0, p)) = (uint16_t)((packed & 0xffu) | ((packed >> 8) & 0xff00u));
        *reinterpret_cast<uint16_t*>(q + plane_byte(e0 + 1u, p)) = (uint16_t)(((packed >> 8) & 0xffu) | ((packed >> 16) & 0xff00u));
    }
    static TM_HD void scalars(uint32_t* units, uint32_t b, int lane, int, float s, float, float, float s32) {
        if (lane == 0) put_scalars(units, b, s * (1.0f / 2048.0f), -8.f * s32);
    }
    template <bool AL> static TM_SD void load(SPtr p, int, uint32_t (&w)[9], Meta& m) {
        load_words<9, AL>(p, w);
        m.d[0] = half_to_float(w[0] & 0xffffu); m.d[1] = half_to_float(w[4] >> 16);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = join16(w[i], w[i + 1]);
    }
    static TM_HD uint32_t code(const uint32_t (&w)[9], int k, int i, int) { return w[(k < 2 ? 0 : 5) + i] & (k & 1 ? 0xF0F0F0F0u : 0x0F0F0F0Fu); }
    static constexpr TM_HD int xw(int k) { return 4 * k; }
    static TM_HD void merge(const int (&c)[4], int, int (&S)[2]) { S[0] = c[0] * 16 + c[1]; S[1] = c[2] * 16 + c[3]; }
    static TM_HD void mask(Meta& m, int nvalid) { mask_d(m.d, nvalid); }
    static TM_HD float combine(const float (&S)[2], const Meta& m, const float4 xs, const float4, float acc) {
        return fma1(m.d[1], fma1(xs.y, S[1], xs.w), fma1(m.d[0], fma1(xs.x, S[0], xs.z), acc));
    }
    TM_LANE_HOST(1)
};

// ---- GGUF Q4_0 (dtype 9): the Q4_0 block with split nibbles, byte j = elements j (low) | j + 16 (high)
// (tensormark/llama.h:4588-4597). Same bytes, same codes: only the elements that they meet differ.
template <> struct Lane<9> : Lane<1> {
    static TM_HD void code_pos(uint32_t e, uint32_t& t, uint32_t& c, uint32_t& byte) {
        t = e >> 6; c = (e & 63u) >> 2; byte = e & 3u;
    }
    static TM_HD uint32_t plane_byte(uint32_t e, int p) { return plane_byte_of<Lane<9>>(e, p); }
    static TM_HD void store_quad(uint32_t* units, uint32_t e0, int p, uint32_t packed) { units[plane_byte(e0, p) >> 2] = packed; }
    TM_LANE_HOST(9)
};

// ---- Q4_1: 20-byte blocks [d:2][m:2][qs:16], byte j = elements j (low) | j+16 (high), w = n*d + m. Sums as for Q4_0.
template <> struct Lane<4> : LanePairs<160, true> {
    static constexpr int UNIT_W = 32, LANE_UNITS = 2, LANE_BYTES = 40;
    static constexpr int NRAW = 10, NACC = 4, MPA = 2;
    struct Meta { float d[2], m[2]; };
    static TM_HD void code_pos(uint32_t e, uint32_t& t, uint32_t& c, uint32_t& byte) { Lane<9>::code_pos(e, t, c, byte); }
    static TM_HD uint32_t plane_byte(uint32_t e, int p) { return plane_byte_of<Lane<4>>(e, p); }
    static TM_HD void store_quad(uint32_t* units, uint32_t e0, int p, uint32_t packed) { units[plane_byte(e0, p) >> 2] = packed; }
    static TM_HD void scalars(uint32_t* units, uint32_t b, int lane, int, float s, float, float, float s32) {
        if (lane == 0) put_scalars(units, b, s * (1.0f / 2048.0f), s32);
    }
    template <bool AL> static TM_SD void load(SPtr p, int, uint32_t (&w)[10], Meta& m) {
        if constexpr (AL) {                                  // a quarter is 40 bytes: 8-byte loads
#pragma unroll
            for (int i = 0; i < 5; ++i) { const uint2 v = ld8(p + 8 * i); w[2 * i] = v.x; w[2 * i + 1] = v.y; }
        } else {
            load_words<10, AL>(p, w);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) { m.d[h] = half_to_float(w[5 * h] & 0xffffu); m.m[h] = half_to_float(w[5 * h] >> 16); }
    }
    static TM_HD uint32_t code(const uint32_t (&w)[10], int k, int i, int) { return w[(k < 2 ? 1 : 6) + i] & (k & 1 ? 0xF0F0F0F0u : 0x0F0F0F0Fu); }
    static constexpr TM_HD int xw(int k) { return 4 * k; }
    static TM_HD void merge(const int (&c)[4], int, int (&S)[2]) { S[0] = c[0] * 16 + c[1]; S[1] = c[2] * 16 + c[3]; }
    static TM_HD void mask(Meta& m, int nvalid) { mask_d(m.d, nvalid); mask_d(m.m, nvalid); }
    static TM_HD float combine(const float (&S)[2], const Meta& m, const float4 xs, const float4, float acc) {
        acc += fma1(m.d[0] * xs.x, S[0], m.m[0] * xs.z);
        return acc + fma1(m.d[1] * xs.y, S[1], m.m[1] * xs.w);
    }
    TM_LANE_HOST(4)
};

// Sub-blocks 2t, 2t + 1 of a Q4_K / Q5_K super-block: d * scale and dmin * min of both (quant.h:256-264).
struct MetaK { float d[2], m[2]; };
TM_HD void k_scales(const uint32_t (&h)[4], int t, MetaK& m) {
    const float d = half_to_float(h[0] & 0xffffu), dmin = half_to_float(h[0] >> 16);
    // pairs j = 2t, 2t + 1 are neighbouring bytes of each of the three scale words
    const uint32_t sh = 16u * ((uint32_t)t & 1u);
    const uint32_t a = (h[1] >> sh) & 0xffffu, b = (h[2] >> sh) & 0xffffu, c = (h[3] >> sh) & 0xffffu;
    const bool low = t < 2;
    const uint32_t s = low ? a & 0x3F3Fu : (c & 0x0F0Fu) | ((a >> 2) & 0x3030u);
    const uint32_t n = low ? b & 0x3F3Fu : ((c >> 4) & 0x0F0Fu) | ((b >> 2) & 0x3030u);
    m.d[0] = d * (float)(s & 0xffu); m.d[1] = d * (float)(s >> 8);
    m.m[0] = dmin * (float)(n & 0xffu); m.m[1] = dmin * (float)(n >> 8);
}

// ---- Q5_K: 176-byte super-blocks of 256: quarter t = the 32 bytes qs[32t..], low nibbles sub-block 2t, high 2t + 1,
// fifth bits in bit 2t / 2t + 1 of qh[0..31]. Sums: low nibbles, 16 x high nibbles, 2^2t x the fifth bits of sub-block 2t,
// 2^(2t+1) x those of 2t + 1; the second result is 16 times the sub-block's.
template <> struct Lane<5> : LanePairs<176, true> {
    static constexpr int UNIT_W = 256, LANE_UNITS = 1, LANE_BYTES = 0;
    static constexpr int NRAW = 16, NACC = 4, MPA = 4;
    using Meta = MetaK;
    static TM_HD void code_pos(uint32_t e, uint32_t& t, uint32_t& c, uint32_t& byte) { Lane<0>::code_pos(e, t, c, byte); }
    static TM_HD uint32_t plane_byte(uint32_t e, int p) { return plane_byte_of<Lane<5>>(e, p); }
    static TM_HD void store_quad(uint32_t* units, uint32_t e0, int p, uint32_t packed) { units[plane_byte(e0, p) >> 2] = packed; }
    static TM_HD void scalars(uint32_t* units, uint32_t b, int lane, int, float s, float, float, float s32) {
        if (lane == 0) put_scalars(units, b, s * (b & 1u ? 1.0f / 2048.0f : 1.0f / 128.0f), s32);
    }
    template <bool AL> static TM_SD void load16(SPtr p, uint32_t* w) {
        uint32_t v[4];
        if constexpr (AL) { const uint4 q = ld16(p); v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }
        else load_words<4, false>(p, v);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = v[i];
    }
    template <bool AL> static TM_SD void load(SPtr p, int t, uint32_t (&w)[16], Meta& m) {
        uint32_t hdr[4];
        load16<AL>(p, hdr);
        load16<AL>(p + 48 + 32 * t, w); load16<AL>(p + 64 + 32 * t, w + 4);
        load16<AL>(p + 16, w + 8); load16<AL>(p + 32, w + 12);
        k_scales(hdr, t, m);
    }
    static TM_HD uint32_t code(const uint32_t (&w)[16], int k, int i, int t) {
        if (k < 2) return w[i] & (k ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
        return w[8 + i] & (k == 2 ? 0x01010101u << (2 * t) : 0x02020202u << (2 * t));
    }
    static constexpr TM_HD int xw(int k) { return 8 * (k & 1); }
    static TM_HD void merge(const int (&c)[4], int t, int (&S)[2]) {
        S[0] = c[0] + (c[2] >> (2 * t)) * 16;                // the shifts are exact: every term has the factor
        S[1] = c[1] + (c[3] >> (2 * t + 1)) * 256;
    }
    static TM_HD void mask(Meta&, int) {}                    // rows are whole super-blocks
    static TM_HD float combine(const float (&S)[2], const Meta& m, const float4 xs, const float4, float acc) {
        acc = fma1(m.d[0] * xs.x, S[0], fma1(-m.m[0], xs.z, acc));
        return fma1(m.d[1] * xs.y, S[1], fma1(-m.m[1], xs.w, acc));
    }
    TM_LANE_HOST(5)
};

// ---- Q4_K: 144-byte super-blocks of 256 (tensormark/quant.h:222-228, 282-301): the Q5_K block without the high bits.
template <> struct Lane<8> : Lane<5> {
    static constexpr int GB = 144, STEP_BYTES = 8 * 144, NRAW = 8, NACC = 2;
    template <bool AL> static TM_SD void load(SPtr p, int t, uint32_t (&w)[8], Meta& m) {
        uint32_t hdr[4];
        load16<AL>(p, hdr);
        load16<AL>(p + 16 + 32 * t, w); load16<AL>(p + 32 + 32 * t, w + 4);
        k_scales(hdr, t, m);
    }
    static TM_HD uint32_t code(const uint32_t (&w)[8], int k, int i, int) { return w[i] & (k ? 0xF0F0F0F0u : 0x0F0F0F0Fu); }
    static TM_HD void merge(const int (&c)[2], int, int (&S)[2]) { S[0] = c[0]; S[1] = c[1]; }
    TM_LANE_HOST(8)
};

// ---- Q6_K: 210-byte super-blocks of 256, only 2-byte aligned. Quarter t = half h = t / 2, weights l in [16u, 16u + 16)
// with u = t % 2, of the four runs j (elements 128h + 32j + l): 16 bytes of ql for j even / odd, 16 of qh, one int8
// sub-scale per run; the sum term of a run is -32 sum(x). Sums per run: its nibbles (16 x for j = 2, 3) and 4^j x its high
// bit pairs. Thread t takes the four words of its 16-byte pieces in the
// order t, t + 1, ... (mod 4): the quarters of a row start a multiple of 16 bytes apart and would otherwise meet in
// the same shared-memory banks.
template <> struct Lane<6> {
    static constexpr int GB = 210, NR = 4, NRAW = 12, NACC = 8, MPA = 2;
    static constexpr bool SIGNED = false;
    static constexpr int STEP_W = 2048, STEP_BYTES = 1680, UNIT_W = 256, LANE_UNITS = 1, LANE_BYTES = 0, XW = kXGroupWords / 4;
    static constexpr bool NEEDS_SUMS = true;
    struct X { uint32_t w[XW]; };
    struct Meta { float d, s[4]; };
    static TM_HD void code_pos(uint32_t e, uint32_t& t, uint32_t& c, uint32_t& byte) {
        const uint32_t j = (e >> 5) & 3u, l = e & 31u;
        t = 2u * (e >> 7) + (l >> 4);
        c = 4u * j + ((((l & 15u) >> 2) - t) & 3u); byte = l & 3u;
    }
    static TM_HD uint32_t plane_byte(uint32_t e, int p) { return plane_byte_of<Lane<6>>(e, p); }
    static TM_HD void store_quad(uint32_t* units, uint32_t e0, int p, uint32_t packed) { units[plane_byte(e0, p) >> 2] = packed; }
    static TM_HD void scalars(uint32_t* units, uint32_t b, int lane, int, float s, float, float s16, float) {
        if (lane & 15) return;                               // lanes 0 and 16 hold the sums of the two 16-runs, one per quarter of the half
        uint32_t* f = units + (b >> 3) * (uint32_t)kXGroupWords + 128u + 16u * ((b & 7u) >> 2) + 8u * (uint32_t)(lane >> 4) + (b & 3u);
        f[0] = as_uint(s * (b & 2u ? 1.0f / 2048.0f : 1.0f / 128.0f));
        f[4] = as_uint(-32.f * s16);
    }
    template <bool AL> static TM_SD void load(SPtr p, int t, uint32_t (&v)[12], Meta& m) {
        const int h = t >> 1, u = t & 1;
        const SPtr run[3] = {p + 64 * h + 16 * u, p + 64 * h + 32 + 16 * u, p + 128 + 32 * h + 16 * u};
        const uint32_t mis = odd_half(p);                    // the same for the whole warp when rows are 16-byte aligned
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int w = 4 * ((i + t) & 3) - (int)mis;
#pragma unroll
            for (int k = 0; k < 3; ++k) v[4 * k + i] = ld4(run[k] + w);
            if (!AL || mis) {
#pragma unroll
                for (int k = 0; k < 3; ++k) v[4 * k + i] = funnel_r(v[4 * k + i], mis ? ld4(run[k] + w + 4) : 0u, mis * 8u);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) m.s[j] = (float)(int8_t)(ld2(p + 192 + 8 * h + 2 * j) >> (8 * u));
        m.d = half_to_float(ld2(p + 208));
    }
    static TM_HD uint32_t code(const uint32_t (&v)[12], int k, int i, int) {
        const int j = k >> 1;
        if (k & 1) return v[8 + i] & (0x03030303u << (2 * j));
        return v[4 * (j & 1) + i] & (j < 2 ? 0x0F0F0F0Fu : 0xF0F0F0F0u);
    }
    static constexpr TM_HD int xw(int k) { return 4 * (k >> 1); }
    static TM_HD void merge(const int (&c)[8], int, int (&S)[4]) {
        S[0] = c[0] + c[1] * 16; S[1] = c[2] + c[3] * 4; S[2] = c[4] + c[5] * 16; S[3] = c[6] + c[7] * 4;
    }
    static TM_HD void mask(Meta&, int) {}
    static TM_HD float combine(const float (&S)[4], const Meta& m, const float4 xs, const float4 xz, float acc) {
        float v = m.s[0] * fma1(xs.x, S[0], xz.x);
        v = fma1(m.s[1], fma1(xs.y, S[1], xz.y), v);
        v = fma1(m.s[2], fma1(xs.z, S[2], xz.z), v);
        v = fma1(m.s[3], fma1(xs.w, S[3], xz.w), v);
        return fma1(m.d, v, acc);
    }
    TM_LANE_HOST(6)
};

// Offset of quarter t inside a row's group (the K-quants' quarters share a super-block: offset 0).
template <int DT> TM_HD uint32_t quarter_off(uint32_t t) { return Lane<DT>::LANE_UNITS == 2 ? t * (uint32_t)Lane<DT>::LANE_BYTES : 0u; }

#if defined(__CUDACC__)
// D = A B (+ D), A unsigned or signed bytes, B signed.
template <bool SIGNED, bool FIRST>
__device__ __forceinline__ void mma_i8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
#define TM_MMA(T) "mma.sync.aligned.m16n8k32.row.col.s32." T ".s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
    if constexpr (FIRST) {
        if constexpr (SIGNED)
            asm volatile(TM_MMA("s8") "{%10,%10,%10,%10};" : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
        else
            asm volatile(TM_MMA("u8") "{%10,%10,%10,%10};" : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
    } else {
        if constexpr (SIGNED)
            asm volatile(TM_MMA("s8") "{%0,%1,%2,%3};" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        else
            asm volatile(TM_MMA("u8") "{%0,%1,%2,%3};" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
#undef TM_MMA
}
// A thread's share of one group of x. xb: where it reads its B operand - the group's image at its column when the
// column's quarter is this thread's k range, a group of zeros otherwise; xf: its quarter's eight floats.
struct XRegs { uint4 b[4]; float4 xs, xz; };
__device__ __forceinline__ float4 ld_f4(SPtr p) { const uint4 v = ld16(p); return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
template <int DT, bool FINE> __device__ __forceinline__ void load_x(XRegs& x, SPtr xb, SPtr xf) {
#pragma unroll
    for (int k = 0; k < 4; ++k) if (!FINE) x.b[k] = ld16(xb + 128 * k);
    x.xs = ld_f4(xf);
    if (Lane<DT>::NR == 4) x.xz = ld_f4(xf + 16);
}
// Quarter t of rows g (r0: the quarter's bytes, quarter_off) and g + 8 (r1) of the tile times one group: their two
// partial sums. nvalid: 32-blocks of this quarter that exist (2, but for the last group of a row that is no multiple of
// 256). FINE: four planes of x, the B operands at xb and, of the second pair, at fine (registers are too few to hold them).
template <int DT, bool AL, bool FINE>
__device__ __forceinline__ void group_dot(SPtr r0, SPtr r1, const XRegs& x, SPtr xb, SPtr fine, int t, int nvalid, float& acc0, float& acc1) {
    using L = Lane<DT>;
    uint32_t w0[L::NRAW], w1[L::NRAW];
    typename L::Meta m0, m1;
    L::template load<AL>(r0, t, w0, m0);
    L::template load<AL>(r1, t, w1, m1);
    float f0[L::NR], f1[L::NR];
    auto planes = [&](auto operand, bool rest) {             // operand(i): B words of MMA pair i (two MMAs)
        int s0[L::NACC], s1[L::NACC], S0[L::NR], S1[L::NR];
#pragma unroll
        for (int k = 0; k < L::NACC; ++k) {
            int c[4];
#pragma unroll
            for (int i = 0; i < L::MPA; ++i) {
                const uint4 b = operand((L::xw(k) + 2 * i) / 4);
                const uint32_t b0 = i & 1 ? b.z : b.x, b1 = i & 1 ? b.w : b.y;      // xw(k) is a multiple of 4
                const uint32_t p = L::code(w0, k, 2 * i, t), q = L::code(w1, k, 2 * i, t), r = L::code(w0, k, 2 * i + 1, t), s = L::code(w1, k, 2 * i + 1, t);
                if (i == 0) mma_i8<L::SIGNED, true>(c, p, q, r, s, b0, b1);
                else mma_i8<L::SIGNED, false>(c, p, q, r, s, b0, b1);
            }
            s0[k] = c[0] * 128 + c[1]; s1[k] = c[2] * 128 + c[3];
        }
        L::merge(s0, t, S0);
        L::merge(s1, t, S1);
#pragma unroll
        for (int r = 0; r < L::NR; ++r) {
            f0[r] = rest ? fmaf((float)S0[r], 1.0f / 16384.0f, f0[r]) : (float)S0[r];
            f1[r] = rest ? fmaf((float)S1[r], 1.0f / 16384.0f, f1[r]) : (float)S1[r];
        }
    };
    if constexpr (FINE) {
        planes([&](int i) { return ld16(xb + 128 * i); }, false);
        planes([&](int i) { return ld16(fine + 128 * i); }, true);
    } else {
        planes([&](int i) { return x.b[i]; }, false);
    }
    if (nvalid < 2) { L::mask(m0, nvalid); L::mask(m1, nvalid); }
    acc0 = L::combine(f0, m0, x.xs, x.xz, 0.f);
    acc1 = L::combine(f1, m1, x.xs, x.xz, 0.f);
}
#else
// What thread t of a row computes, without the tensor core.
template <int DT> float LaneHost<DT>::dot(const uint8_t* quarter, const uint32_t* w, int t, int nvalid) {
    using L = Lane<DT>;
    uint32_t raw[L::NRAW];
    typename L::Meta m;
    L::template load<false>(quarter, t, raw, m);
    if (nvalid < 2) L::mask(m, nvalid);
    int c[L::NACC], S[L::NR];
    for (int k = 0; k < L::NACC; ++k) {
        c[k] = 0;
        for (int i = 0; i < 2 * L::MPA; ++i) {
            const uint32_t v = L::code(raw, k, i, t);
            for (int p = 0; p < 2; ++p) c[k] += (p ? 1 : 128) * (L::SIGNED ? dp4a_ss(v, w[16 * p + L::xw(k) + i], 0) : dp4a_us(v, w[16 * p + L::xw(k) + i], 0));
        }
    }
    L::merge(c, t, S);
    float f[L::NR];
    for (int r = 0; r < L::NR; ++r) f[r] = (float)S[r];
    const float4 xs = {as_float(w[32]), as_float(w[33]), as_float(w[34]), as_float(w[35])};
    const float4 xz = {as_float(w[36]), as_float(w[37]), as_float(w[38]), as_float(w[39])};
    return L::combine(f, m, xs, xz, 0.f);
}
// The x words of quarter u % 4 of group u / 4 in MMA order: plane 0, plane 1, then the eight floats.
template <int DT> void load_x_unit(typename Lane<DT>::X& x, const uint32_t* units, uint32_t u) {
    for (uint32_t p = 0; p < 2; ++p)
        for (uint32_t c = 0; c < 16; ++c) x.w[16 * p + c] = units[x_word(u >> 2, u & 3u, c, p)];
    for (uint32_t i = 0; i < 8; ++i) x.w[32 + i] = units[(u >> 2) * (uint32_t)kXGroupWords + 128u + 8u * (u & 3u) + i];
}
#endif

}  // namespace tmc
