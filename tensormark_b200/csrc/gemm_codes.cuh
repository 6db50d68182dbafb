// gemm_codes.cuh — a row's serialized blocks -> fp16 pairs in registers, for the GEMM that keeps no fp16 copy of its weights.
//
// Codes<DT>::stage<S>() turns stage S (64 weights of a group of 256, S = 0..3) of one row into 32 registers of two fp16
// each. Within a group the weights come out in whatever order costs fewest instructions (a nibble word w gives the pairs
// w, w >> 4, w >> 8, w >> 12, masked); k_of() names the weight at each place and the activations are laid out to match.
// Every value is the dequantizer's fp32 result rounded once to fp16:
//   * Q4_0, GGUF Q4_0, Q8_0: code * d in half arithmetic: the code is exact in fp16, so the product is rounded once.
//   * Q4_1: one half fma (n d + m rounded once; the fp32 form rounds twice).
//   * K-quants: fp32 products (exact: at most 24 significant bits), fp32 subtraction of the minimum, one rounding.
#pragma once

#include "common.cuh"

#include <cuda_fp16.h>

namespace tmc {

__device__ __forceinline__ uint4 lds_line(uint32_t p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p));
    return v;
}
template <int L> __device__ __forceinline__ void lds_lines(uint32_t p, uint32_t (&v)[4 * L]) {
#pragma unroll
    for (int i = 0; i < L; ++i) {
        const uint4 q = lds_line(p + 16u * i);
        v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
    }
}
// the 32-bit word at byte B (even) of a register array
template <int B, int NV> __device__ __forceinline__ uint32_t word_at(const uint32_t (&v)[NV]) {
    if constexpr (B % 4 == 0) return v[B / 4];
    else return __funnelshift_r(v[B / 4], v[B / 4 + 1], 16);
}
template <int B, int NV> __device__ __forceinline__ uint32_t half_twice(const uint32_t (&v)[NV]) {      // the half at byte B, in both halves
    return __byte_perm(v[B / 4], 0, B % 4 ? 0x3232 : 0x1010);
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
template <uint32_t MASK> __device__ __forceinline__ uint32_t magic(uint32_t w) { return (w & MASK) | 0x64006400u; }    // 1024 + code in each half
__device__ __forceinline__ uint32_t scaled(uint32_t m, uint32_t bias, uint32_t d) { return as_u32(__hmul2(__hsub2(as_h2(m), as_h2(bias)), as_h2(d))); }
// Codes 0..63 in the bytes of `u`, each with bit 7 set: a byte permutation makes the float 1 + code / 128 of one, and an
// fma takes the code out of it again, so no conversion instruction (half rate, two per pair) is needed. scale * (code - BIAS)
// is exact in fp32 (scale: at most 18 bits), MIN subtracts a minimum with one rounding. o[at], o[at + 1]: bytes 0, 1 and 2, 3.
template <int BIAS, bool MIN> __device__ __forceinline__ void scaled_f32(uint32_t u, float scale, float minimum, uint32_t (&o)[32], int at) {
    const float a = 128.0f * scale, b = -(float)(128 + BIAS) * scale;
    float f[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[i] = __fmaf_rn(__uint_as_float(__byte_perm(u, 0x3f000000u, 0x7044 | (i << 8))), a, b);
        if constexpr (MIN) f[i] = __fsub_rn(f[i], minimum);
    }
    o[at] = as_u32(__floats2half2_rn(f[0], f[1]));
    o[at + 1] = as_u32(__floats2half2_rn(f[2], f[3]));
}
template <uint32_t MASK, uint32_t OR> __device__ __forceinline__ uint32_t and_or(uint32_t w) { return (w & MASK) | OR; }
__device__ __forceinline__ float half_lo(uint32_t v) { return __low2float(as_h2(v)); }
__device__ __forceinline__ float half_hi(uint32_t v) { return __high2float(as_h2(v)); }

// L lines from byte `off` (0..15) of the line at p on: what a row that does not begin on a 16-byte boundary needs.
template <int L, int NV = 4 * L> __device__ __forceinline__ void lds_shifted(uint32_t p, uint32_t off, uint32_t (&r)[NV]) {
    constexpr int NL = (NV + 3) / 4 + 1;
    uint32_t v[4 * NL], u[NV + 2], t[NV + 1];
    lds_lines<NL>(p, v);
#pragma unroll
    for (int i = 0; i < NV + 2; ++i) u[i] = (off & 8u) ? v[i + 2 < 4 * NL ? i + 2 : 4 * NL - 1] : v[i];
#pragma unroll
    for (int i = 0; i < NV + 1; ++i) t[i] = (off & 4u) ? u[i + 1] : u[i];
#pragma unroll
    for (int i = 0; i < NV; ++i) r[i] = __funnelshift_r(t[i], t[i + 1], 8u * (off & 3u));
}
template <bool AL, int L> __device__ __forceinline__ void row_lines(uint32_t p, uint32_t off, uint32_t (&v)[4 * L]) {
    if constexpr (AL) lds_lines<L>(p, v);
    else lds_shifted<L>(p, off, v);
}

// kBytes: serialized bytes of a group of 256 weights; `row` is the line that a row's group begins in, `off` bytes further
// on (AL: the group begins on the line, or `off` is not looked at for other reasons).
template <int DT> struct Codes;

struct Block32Codes {                                      // 4-bit blocks of 32: a half scale, then 16 code bytes
    // byte j of a Q4_0 block holds weights 2j and 2j + 1; of a GGUF Q4_0 or Q4_1 block weights j and j + 16
    template <bool ADJACENT> static __host__ __device__ constexpr int k_of(int s, int i) {
        const int reg = i >> 1, hi = i & 1, w = reg >> 2, t = reg & 3;
        return 64 * s + 32 * (w >> 2) + (ADJACENT ? 8 * (w & 3) + t + 4 * hi : 4 * (w & 3) + 2 * hi + (t >> 1) + 16 * (t & 1));
    }
};
template <> struct Codes<1> {                              // Q4_0
    static constexpr uint32_t kBytes = 144;
    static __host__ __device__ constexpr int k_of(int s, int i) { return Block32Codes::k_of<true>(s, i); }
    template <int S, bool AL> static __device__ __forceinline__ void stage(uint32_t row, uint32_t off, uint32_t (&o)[32]) {
        constexpr int B = 36 * S, LO = B & 15;
        uint32_t v[12];
        row_lines<AL, 3>(row + (B & ~15), off, v);
        blocks<LO>(v, o);
    }
    template <int LO> static __device__ __forceinline__ void blocks(const uint32_t (&v)[12], uint32_t (&o)[32]) {
        nibbles(half_twice<LO>(v), word_at<LO + 2>(v), o, 0);
        nibbles(half_twice<LO>(v), word_at<LO + 6>(v), o, 4);
        nibbles(half_twice<LO>(v), word_at<LO + 10>(v), o, 8);
        nibbles(half_twice<LO>(v), word_at<LO + 14>(v), o, 12);
        nibbles(half_twice<LO + 18>(v), word_at<LO + 20>(v), o, 16);
        nibbles(half_twice<LO + 18>(v), word_at<LO + 24>(v), o, 20);
        nibbles(half_twice<LO + 18>(v), word_at<LO + 28>(v), o, 24);
        nibbles(half_twice<LO + 18>(v), word_at<LO + 32>(v), o, 28);
    }
    static __device__ __forceinline__ void nibbles(uint32_t d, uint32_t w, uint32_t (&o)[32], int at) {
        o[at] = scaled(magic<0x000f000fu>(w), 0x64086408u, d);
        o[at + 1] = scaled(magic<0x000f000fu>(w >> 4), 0x64086408u, d);
        o[at + 2] = scaled(magic<0x000f000fu>(w >> 8), 0x64086408u, d);
        o[at + 3] = scaled(magic<0x000f000fu>(w >> 12), 0x64086408u, d);
    }
};
template <> struct Codes<9> : Codes<1> {                   // GGUF Q4_0: the same bytes, weights j and j + 16 in byte j
    static __host__ __device__ constexpr int k_of(int s, int i) { return Block32Codes::k_of<false>(s, i); }
};
template <> struct Codes<4> {                              // Q4_1: d, m, 16 code bytes
    static constexpr uint32_t kBytes = 160;
    static __host__ __device__ constexpr int k_of(int s, int i) { return Block32Codes::k_of<false>(s, i); }
    template <int S, bool AL> static __device__ __forceinline__ void stage(uint32_t row, uint32_t off, uint32_t (&o)[32]) {
        constexpr int B = 40 * S, LO = (B & 15) / 4;
        uint32_t v[12];
        row_lines<AL, 3>(row + (B & ~15), off, v);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t dm = v[LO + 5 * b], d = __byte_perm(dm, 0, 0x1010), m = __byte_perm(dm, 0, 0x3232);
#pragma unroll
            for (int w = 0; w < 4; ++w)
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    o[16 * b + 4 * w + t] = as_u32(__hfma2(__hsub2(as_h2(magic<0x000f000fu>(v[LO + 5 * b + 1 + w] >> (4 * t))), as_h2(0x64006400u)), as_h2(d), as_h2(m)));
        }
    }
};
template <> struct Codes<0> {                              // Q8_0: d, 32 signed codes
    static constexpr uint32_t kBytes = 272;
    static __host__ __device__ constexpr int k_of(int s, int i) { return 64 * s + i; }
    template <int S, bool AL> static __device__ __forceinline__ void stage(uint32_t row, uint32_t off, uint32_t (&o)[32]) {
        constexpr int B = 68 * S, LO = B & 15;
        uint32_t v[20];
        row_lines<AL, 5>(row + (B & ~15), off, v);
        words<LO + 2>(v, half_twice<LO>(v), o, 0);
        words<LO + 36>(v, half_twice<LO + 34>(v), o, 16);
    }
    template <int B> static __device__ __forceinline__ void words(const uint32_t (&v)[20], uint32_t d, uint32_t (&o)[32], int at) {
        one(word_at<B>(v), d, o, at); one(word_at<B + 4>(v), d, o, at + 2); one(word_at<B + 8>(v), d, o, at + 4); one(word_at<B + 12>(v), d, o, at + 6);
        one(word_at<B + 16>(v), d, o, at + 8); one(word_at<B + 20>(v), d, o, at + 10); one(word_at<B + 24>(v), d, o, at + 12); one(word_at<B + 28>(v), d, o, at + 14);
    }
    static __device__ __forceinline__ void one(uint32_t w, uint32_t d, uint32_t (&o)[32], int at) {
        const uint32_t u = w ^ 0x80808080u;                                   // code + 128
        o[at] = scaled(__byte_perm(u, 0x64646464u, 0x4140), 0x64806480u, d);
        o[at + 1] = scaled(__byte_perm(u, 0x64646464u, 0x4342), 0x64806480u, d);
    }
};
// The header of a Q4_K or Q5_K super-block -> d * scale and dmin * minimum of sub-blocks 2S and 2S + 1 (tensormark/quant.h:282-330).
template <int S> __device__ __forceinline__ void k_scales(const uint4 h, float (&a)[2], float (&b)[2]) {
    const float d = half_lo(h.x), dm = half_hi(h.x);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int j = 2 * S + c;
        uint32_t s6, m6;
        if (j < 4) { s6 = (h.y >> (8 * j)) & 63u; m6 = (h.z >> (8 * j)) & 63u; }
        else {
            const int r = 8 * (j - 4);
            s6 = ((h.w >> r) & 15u) | (((h.y >> (r + 6)) & 3u) << 4);
            m6 = ((h.w >> (r + 4)) & 15u) | (((h.z >> (r + 6)) & 3u) << 4);
        }
        a[c] = __fmul_rn(d, __uint2float_rn(s6));
        b[c] = __fmul_rn(dm, __uint2float_rn(m6));
    }
}
struct KCodes {                                            // registers 4w + 2c, + 1: bytes 4w .. 4w + 3 of sub-block c
    static __host__ __device__ constexpr int k_of(int s, int i) { return 64 * s + 32 * ((i >> 2) & 1) + 4 * (i >> 3) + (i & 3); }
};
template <> struct Codes<8> : KCodes {                     // Q4_K
    static constexpr uint32_t kBytes = 144;
    template <int S, bool AL> static __device__ __forceinline__ void stage(uint32_t row, uint32_t off, uint32_t (&o)[32]) {
        uint32_t v[8];
        static_assert(AL, "");
        lds_lines<2>(row + 16 + 32 * S, v);
        float a[2], b[2];
        k_scales<S>(lds_line(row), a, b);
#pragma unroll
        for (int w = 0; w < 8; ++w)
#pragma unroll
            for (int c = 0; c < 2; ++c) scaled_f32<0, true>(and_or<0x0f0f0f0fu, 0x80808080u>(v[w] >> (4 * c)), a[c], b[c], o, 4 * w + 2 * c);
    }
};
template <> struct Codes<5> : KCodes {                     // Q5_K
    static constexpr uint32_t kBytes = 176;
    template <int S, bool AL> static __device__ __forceinline__ void stage(uint32_t row, uint32_t off, uint32_t (&o)[32]) {
        uint32_t v[8], q[8];
        static_assert(AL, "");
        lds_lines<2>(row + 48 + 32 * S, v);
        lds_lines<2>(row + 16, q);
        float a[2], b[2];
        k_scales<S>(lds_line(row), a, b);
#pragma unroll
        for (int w = 0; w < 8; ++w)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                constexpr int up = 4 - 2 * S;                                 // brings bit 2 S + c of a byte to bit 4
                const int sh = up - c;
                const uint32_t hb = (sh >= 0 ? q[w] << (sh & 31) : q[w] >> (-sh & 31)) & 0x10101010u;
                scaled_f32<0, true>(and_or<0x0f0f0f0fu, 0x80808080u>(v[w] >> (4 * c)) | hb, a[c], b[c], o, 4 * w + 2 * c);
            }
    }
};
template <> struct Codes<6> {                              // Q6_K: 210 bytes, so `off` counts in every case
    static constexpr uint32_t kBytes = 210;
    static __host__ __device__ constexpr int k_of(int s, int i) {      // registers 8w + 2j, + 1: bytes 4w .. 4w + 3 of sub-block j
        return 128 * (s >> 1) + 32 * ((i >> 2) & 3) + 16 * (s & 1) + 4 * (i >> 4) + (i & 3);
    }
    template <int S, bool> static __device__ __forceinline__ void stage(uint32_t row, uint32_t off, uint32_t (&o)[32]) {
        constexpr int H = S >> 1, L = S & 1;
        float ds[4];
        {
            uint32_t sc[4], dw[1];
            lds_shifted<1>(row + 192, off, sc);                    // 16 scales
            lds_shifted<1, 1>(row + 208, off, dw);
            const float d = half_lo(dw[0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                constexpr int at = 8 * H + L;
                const int byte = at + 2 * j;
                ds[j] = __fmul_rn(d, __int2float_rn((int)(int8_t)(sc[byte / 4] >> (8 * (byte % 4)))));
            }
        }
        uint32_t q0[4], q1[4], qh[4];
        lds_shifted<1>(row + 64 * H + 16 * L, off, q0);
        lds_shifted<1>(row + 64 * H + 32 + 16 * L, off, q1);
        lds_shifted<1>(row + 128 + 32 * H + 16 * L, off, qh);
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t nib = and_or<0x0f0f0f0fu, 0x80808080u>((j & 1 ? q1[w] : q0[w]) >> (j & 2 ? 4 : 0));
                const uint32_t hb = (j == 3 ? qh[w] >> 2 : qh[w] << (j == 3 ? 0 : 4 - 2 * j)) & 0x30303030u;
                scaled_f32<32, false>(nib | hb, ds[j], 0.f, o, 8 * w + 2 * j);
            }
    }
};

}  // namespace tmc
