// gemv_f16.cu — y = W x for tensors that a container keeps as plain 16-bit rows (fp16, dtype 3; bf16, dtype 10), the
// embedding-row gather from such a table, and the in-place nibble reorder that turns GGUF's Q4_0 blocks into the
// container's.
//
// Replaces the reference's f16_gemv_coop_r1/2/4 (tensormark/metal.h:575-613, host side tok_gemv_h 3693-3721) and
// embed_h_row (2396-2407, tok_embed_h 3260-3271); bf16 has no GPU kernel in the reference (its loader keeps such
// tensors on the CPU, tensormark/llama.h:4599-4606) and is served by the same kernel here.
//
// Bound: HBM, 2 bytes per weight. x is copied into shared memory once per CTA as fp32; LPR lanes (8, or 1 to 8 warps) share
// a row and read it as 16-byte pieces (eight weights), eight independent loads in flight per lane, fp32 FMA, one shuffle
// reduction per warp and row (how many lanes share a row depends on N, and with it the last bits of its sum).
//   * A CTA's first loads do not depend on x: where the weights are the lane's registered ones, they are requested before
//     x is waited for. A caller's own device weights may come from the kernel before, as x may: before the wait they are
//     only asked into L2, and requested while x is on its way into shared memory (2000 x 2048 3.9 us a launch with the
//     early request, 4.1 so, 4.9 without the prefetch and behind x; 4096 x 4096 9.4, 9.8, 11.4).
//   * Few rows take more warps each, so that the machine is not left with one row per SM and a chain of loads (105 x 3584:
//     6.8 us a launch with one, now 3.4; 43913 x 4896: 82.7 us, now 78.6).
// Rows must be 16-byte aligned for that form (K a multiple of 8 and an aligned base); anything else takes a scalar-load
// kernel.
#include "common.cuh"

#include <cuda_fp16.h>
#include <type_traits>

namespace tmc {
namespace {

template <bool BF16> __device__ __forceinline__ float2 pair_to_float(uint32_t u) {
    if constexpr (BF16) return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
    else return __half22float2(*reinterpret_cast<const __half2*>(&u));
}
template <bool BF16> __device__ __forceinline__ float one_to_float(uint16_t h) {
    if constexpr (BF16) return __uint_as_float((uint32_t)h << 16);
    else return __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <bool BF16> __device__ __forceinline__ float dot8(const uint4 w, const float* xs) {
    const float4 a = *reinterpret_cast<const float4*>(xs), b = *reinterpret_cast<const float4*>(xs + 4);
    const float2 p0 = pair_to_float<BF16>(w.x), p1 = pair_to_float<BF16>(w.y), p2 = pair_to_float<BF16>(w.z), p3 = pair_to_float<BF16>(w.w);
    float s = p0.x * a.x;
    s = fmaf(p0.y, a.y, s); s = fmaf(p1.x, a.z, s); s = fmaf(p1.y, a.w, s);
    s = fmaf(p2.x, b.x, s); s = fmaf(p2.y, b.y, s); s = fmaf(p3.x, b.z, s); s = fmaf(p3.y, b.w, s);
    return s;
}

template <bool BF16, int LPR, bool FIXED>
__global__ void __launch_bounds__(256, 3) gemv_half_rows(const float* x, const uint16_t* W, float* __restrict__ y, uint32_t N, uint32_t K) {
    constexpr uint32_t ROWS = 256 / LPR, STEP = LPR, U = 8, WPR = LPR / 32;    // WPR 0: several rows per warp
    extern __shared__ __align__(16) float xs[];
    __shared__ float sums[2][8];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k8 = K / 8, first = threadIdx.x % LPR;
    uint4 w[U];
    auto request = [&](uint32_t row, uint32_t i0) {
        const uint4* wr = reinterpret_cast<const uint4*>(W + (size_t)row * K);
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
            if (i0 + u * STEP < k8) w[u] = __ldcg(wr + i0 + u * STEP);
    };
    const uint32_t row0 = blockIdx.x * ROWS + threadIdx.x / LPR;
    if (row0 < N) {
        if (FIXED) request(row0, first);
        else if (first == 0)                                    // into L2 only, where a write that is still to come finds them
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(W + (size_t)row0 * K), "r"(min(k8, max(U * STEP, 256u)) * 16u) : "memory");
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");          // x may come from the preceding kernel of the stream
    for (uint32_t i = threadIdx.x; i < K / 4; i += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(xs + 4 * i)), "l"(x + 4 * i) : "memory");
    if (!FIXED && row0 < N) request(row0, first);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    uint32_t turn = 0;
    for (uint32_t base = blockIdx.x * ROWS; base < N; base += gridDim.x * ROWS, turn ^= 1u) {
        const uint32_t row = base + threadIdx.x / LPR, next = row + gridDim.x * ROWS;
        float acc[2] = {0.f, 0.f};
        if (row < N) {
            for (uint32_t i = first; i < k8; i += U * STEP) {
                uint4 v[U];
#pragma unroll
                for (uint32_t u = 0; u < U; ++u) v[u] = w[u];
                if (i + U * STEP < k8) request(row, i + U * STEP);
                else if (next < N) request(next, first);
#pragma unroll
                for (uint32_t u = 0; u < U; ++u)
                    if (i + u * STEP < k8) acc[u & 1] += dot8<BF16>(v[u], xs + 8 * (i + u * STEP));
            }
            if (first >= k8 && next < N) request(next, first);
        }
        float v = acc[0] + acc[1];
#pragma unroll
        for (int o = (LPR < 32 ? LPR : 32) / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if constexpr (WPR > 1) {
            if (lane == 0) sums[turn][warp] = v;
            __syncthreads();                                    // the other half of `sums` is free: everybody has passed this barrier once since
            v = 0.f;
#pragma unroll
            for (uint32_t p = 0; p < WPR; ++p) v += sums[turn][warp / WPR * WPR + p];
        }
        if (first == 0 && row < N) y[row] = v;
    }
}

// any K, any 2-byte aligned base: one warp per row, scalar loads
template <bool BF16>
__global__ void __launch_bounds__(256) gemv_half_generic(const float* x, const uint16_t* __restrict__ W, float* __restrict__ y,
                                                         uint32_t N, uint32_t K) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * 8 + warp;
    if (row >= N) return;
    const uint16_t* wr = W + (size_t)row * K;
    float acc = 0.f;
    for (uint32_t k = lane; k < K; k += 32) acc = fmaf(one_to_float<BF16>(wr[k]), __ldcg(x + k), acc);
    acc = warp_total(acc);
    if (lane == 0) y[row] = acc;
}

// x = row tok[idx] of a 16-bit table (sentinel 0xFFFFFFFF -> zeros), embed_h_row (metal.h:2396-2407)
template <bool BF16>
__global__ void embed_half_row(const uint32_t* tok, uint32_t idx, const uint16_t* __restrict__ W, float* __restrict__ x, uint32_t D) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= D) return;
    const uint32_t row = tok[idx];
    x[k] = row == 0xFFFFFFFFu ? 0.f : one_to_float<BF16>(W[(size_t)row * D + k]);
}

// GGUF Q4_0 (split nibbles: byte j = elements j | j + 16) -> container Q4_0 (byte j = elements 2j | 2j + 1), in place,
// one thread per 18-byte block (tensormark/convert_gguf.cpp:124-135). Scale and codes are unchanged, so the weights are
// bit-identical.
__global__ void q4_split_to_interleaved_kernel(uint8_t* blocks, size_t nblocks) {
    const size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nblocks) return;
    uint8_t* q = blocks + b * 18 + 2;
    uint8_t s[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) s[j] = q[j];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        q[j] = (uint8_t)((s[2 * j] & 15) | ((s[2 * j + 1] & 15) << 4));
        q[j + 8] = (uint8_t)((s[2 * j] >> 4) | ((s[2 * j + 1] >> 4) << 4));
    }
}

}  // namespace

bool launch_gemv_half(const float* x, const void* W, float* y, unsigned N, unsigned K, bool bf16, bool fixed, cudaStream_t st) {
    if (!x || !W || !y) return fail("gemv_h: null pointer");
    if (N == 0) return true;
    if (K == 0) return fail("gemv_h: empty rows");
    if ((uintptr_t)W % 2 || (uintptr_t)x % 4) return fail("gemv_h: misaligned operand");
    const uint16_t* w = (const uint16_t*)W;
    const size_t smem = (size_t)K * 4;
    if (K % 8 == 0 && (uintptr_t)W % 16 == 0 && (uintptr_t)x % 16 == 0 && smem <= 200 * 1024) {
        const unsigned sms = (unsigned)device_sm_count();
        // One wave: three CTAs per SM by registers, fewer where x is long. A row takes as many warps as leave all CTAs in it, with
        // four pieces of the row for every lane (one CTA per SM where x is so long that staging it costs as much as the rows);
        // rows of up to 1024 take eight lanes, so that a lane has as many as it can request, where that fills the machine.
        const unsigned fit = (unsigned)((224 * 1024) / (smem + 2048)), wave = sms * (fit < 1 ? 1 : fit < 3 ? fit : 3);
        unsigned lpr = K <= 1024 && N > 32 * sms ? 8 : 32;
        while (lpr >= 32 && lpr < 256 && (uint64_t)N * lpr * 2 <= 256ull * (smem > 52 * 1024 ? sms : wave) && K / 8 >= 8 * lpr) lpr *= 2;
        // FIXED is part of the kernel's type: as an argument it made the launch 0.35 us longer (24.0 -> 26.8 us for eight small calls).
        auto launch_as = [&](auto b, auto parts, auto f) {
            constexpr auto kernel = gemv_half_rows<decltype(b)::value, decltype(parts)::value, decltype(f)::value>;
            static const cudaError_t attr = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            if (attr != cudaSuccess) return fail("gemv_h: cannot raise the dynamic shared memory limit");
            const unsigned rows = 256 / lpr, want = (N + rows - 1) / rows;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(want < wave ? want : wave); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = smem; cfg.stream = st;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = at; cfg.numAttrs = 1;
            cudaLaunchKernelEx(&cfg, kernel, x, w, y, (uint32_t)N, (uint32_t)K);
            return true;
        };
        auto launch = [&](auto b, auto parts) {
            if constexpr (!decltype(b)::value)                  // the lane's rows are fp16
                if (fixed) return launch_as(b, parts, std::true_type{});
            return launch_as(b, parts, std::false_type{});
        };
        auto pick = [&](auto b) {
            return lpr == 8 ? launch(b, std::integral_constant<int, 8>{}) : lpr == 32 ? launch(b, std::integral_constant<int, 32>{})
                 : lpr == 64 ? launch(b, std::integral_constant<int, 64>{}) : lpr == 128 ? launch(b, std::integral_constant<int, 128>{})
                 : launch(b, std::integral_constant<int, 256>{});
        };
        if (!(bf16 ? pick(std::true_type{}) : pick(std::false_type{}))) return false;
    } else {
        if (bf16) gemv_half_generic<true><<<(N + 7) / 8, 256, 0, st>>>(x, w, y, N, K);
        else gemv_half_generic<false><<<(N + 7) / 8, 256, 0, st>>>(x, w, y, N, K);
    }
    note_launch();
    return check_launch("gemv_h");
}

bool launch_embed_half(const unsigned* tok, unsigned idx, const void* W, float* x, unsigned D, bool bf16, cudaStream_t st) {
    if (!tok || !W || !x || D == 0) return fail("embed_h: bad arguments");
    if (bf16) embed_half_row<true><<<(D + 255) / 256, 256, 0, st>>>(tok, idx, (const uint16_t*)W, x, D);
    else embed_half_row<false><<<(D + 255) / 256, 256, 0, st>>>(tok, idx, (const uint16_t*)W, x, D);
    note_launch();
    return check_launch("embed_h");
}

bool launch_q4_split_to_interleaved(uint8_t* blocks, size_t nblocks, cudaStream_t st) {
    if (!blocks) return fail("q4 repack: null pointer");
    if (nblocks == 0) return true;
    q4_split_to_interleaved_kernel<<<(unsigned)((nblocks + 255) / 256), 256, 0, st>>>(blocks, nblocks);
    note_launch();
    return check_launch("q4 repack");
}

}  // namespace tmc
