// The parts of an encoder layer between its products, on feature-major activations x[features][tokens] (the layout the
// SpMM reads and writes): LayerNorm with the residual sum before it, and softmax attention.  The reference runs both as
// framework operations (end2end/sspmm_e2e/end_to_end.py:44-75).
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>

#include "../../include/sspmm_b200.h"
#include "launch.h"
#include "ptx.cuh"

namespace sspmm_b200 {
namespace enc {

__device__ __forceinline__ void unpack8(const uint4& x, float (&f)[8]) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = v.x; f[2 * i + 1] = v.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 h = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// ---- LayerNorm ------------------------------------------------------------------------------------
// Bound by memory: x (and add) read once, out (and the sum) written once.  A CTA takes TT tokens, as many as give every SM a CTA (8, 16 or
// 32: runs of 16, 32 or 64 bytes), and keeps what it has read for the passes for the mean, the variance and the result in the registers of
// 512 threads; 32 tokens of more than 1024 features go through shared memory.  Through shared memory, 768 x 16384 took 24.0 us,
// with a sum 40.2: every thread added up the warps' sums for itself (64 reads twice), converted every element three times and worked
// on one element per instruction.  From registers, with pairs of elements per instruction and sums that are added up once, 16.6
// and 24.8 (operands that change from call to call); 256 threads with twice the registers take 17.1 and 36.6.  In graph replays 256 x 128 2.75 us
// and 3.19, now 2.28 and 2.63; 768 x 1024 4.68 and 6.15, now 3.77 and 4.77; 512 x 4000 7.36 and 9.83, now 4.10 and 5.14; 3072 x 512 9.25 and
// 15.3, now 7.07 and 11.1.
constexpr int kLnThreads = 256, kLnWideThreads = 512;
__global__ void __launch_bounds__(kLnThreads)
layer_norm_fm_kernel(int hidden, int tokens, const __half* __restrict__ x, const __half* __restrict__ bias, const __half* __restrict__ add,
                     __half* __restrict__ sum_out,
                     const __half* __restrict__ gamma, const __half* __restrict__ beta, float eps, __half* __restrict__ out) {
    constexpr int TT = 32, P = TT / 8, kRows = kLnThreads / P;      // pieces per feature, features per turn
    extern __shared__ uint4 tile[];                         // [hidden][P]
    __shared__ float red[kLnThreads / 32][TT];
    const int piece = threadIdx.x % P, r0 = threadIdx.x / P, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * TT + piece * 8;
    const bool in = t0 < tokens;
    // sum over the features of eight numbers per token, the same in every thread of the piece
    auto total = [&](float (&f)[8]) {
#pragma unroll
        for (int o = P; o < 32; o <<= 1)
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] += __shfl_xor_sync(0xffffffffu, f[e], o);
        if (lane < P)
#pragma unroll
            for (int e = 0; e < 8; ++e) red[warp][piece * 8 + e] = f[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            f[e] = 0.f;
            for (int w = 0; w < kLnThreads / 32; ++w) f[e] += red[w][piece * 8 + e];
        }
        __syncthreads();
    };
    float mean[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int r = r0; r < hidden; r += kRows) {
        uint4 v = make_uint4(0, 0, 0, 0);
        const int64_t at = (int64_t)r * tokens + t0;
        if (in) v = __ldg(reinterpret_cast<const uint4*>(x + at));
        float f[8];
        unpack8(v, f);
        if (bias) {
            const float b = __half2float(__ldg(bias + r));
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __half2float(__float2half_rn(f[e] + b));
            v = pack8(f);
        }
        if (add) {
            float g[8];
            unpack8(in ? __ldg(reinterpret_cast<const uint4*>(add + at)) : make_uint4(0, 0, 0, 0), g);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] += g[e];
            v = pack8(f);
            if (in) *reinterpret_cast<uint4*>(sum_out + at) = v;
            unpack8(v, f);
        }
        tile[r * P + piece] = v;
#pragma unroll
        for (int e = 0; e < 8; ++e) mean[e] += f[e];
    }
    total(mean);
    const float inv = 1.f / (float)hidden;
    float var[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 8; ++e) mean[e] *= inv;
#pragma unroll 4
    for (int r = r0; r < hidden; r += kRows) {
        float f[8];
        unpack8(tile[r * P + piece], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) { const float d = f[e] - mean[e]; var[e] = fmaf(d, d, var[e]); }
    }
    total(var);
#pragma unroll
    for (int e = 0; e < 8; ++e) var[e] = rsqrtf(fmaf(var[e], inv, eps));
#pragma unroll 4
    for (int r = r0; r < hidden; r += kRows) {
        float f[8];
        unpack8(tile[r * P + piece], f);
        const float g = __half2float(gamma[r]), b = __half2float(beta[r]);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = (f[e] - mean[e]) * var[e] * g + b;
        if (in) *reinterpret_cast<uint4*>(out + (int64_t)r * tokens + t0) = pack8(f);
    }
}

// Two fp32 numbers in one register pair; an instruction works on both, each rounded to nearest as by itself.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair_of(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 floats_of(f32x2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ void unpack4(const uint4& x, f32x2 (&f)[4]) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[i] = pair_of(v.x, v.y);
    }
}
__device__ __forceinline__ uint4 pack4(const f32x2 (&f)[4]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = floats_of(f[i]);
        const __half2 h = __floats2half2_rn(v.x, v.y);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// The same with a thread's share in registers: TT tokens, up to 4096 / TT * NV features.
template <int TT, int NV>
__device__ __forceinline__ void layer_norm_tile(int tile, int hidden, int tokens, const __half* __restrict__ x, const __half* __restrict__ bias,
                                                const __half* __restrict__ add, __half* __restrict__ sum_out, const __half* __restrict__ gamma,
                                                const __half* __restrict__ beta, float eps, __half* __restrict__ out) {
    constexpr int P = TT / 8, kRows = kLnWideThreads / P, kPair = NV < 2 ? 1 : 2;
    static_assert(NV % kPair == 0, "whole pairs");
    __shared__ float red[kLnWideThreads / 32][TT];
    __shared__ __align__(16) float whole[2][TT];
    const int piece = threadIdx.x % P, r0 = threadIdx.x / P, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = tile * TT + piece * 8;
    const bool in = t0 < tokens;
    // Sums over the features of eight numbers per token, the same in every thread of the piece.  A lane hands on half of what it has at each
    // step (7 shuffles; 24 with every sum in every lane), and one warp adds up for the CTA.
    auto total = [&](f32x2 (&f)[4], float (&sums)[TT]) {
        f32x2 h[2];
        const bool upper = lane & 16, odd = lane & 8;
#pragma unroll
        for (int e = 0; e < 2; ++e) h[e] = add2(upper ? f[2 + e] : f[e], __shfl_xor_sync(0xffffffffu, upper ? f[e] : f[2 + e], 16));
        const float2 q = floats_of(add2(odd ? h[1] : h[0], __shfl_xor_sync(0xffffffffu, odd ? h[0] : h[1], 8)));
        const float own = lane & 4 ? q.y : q.x, other = lane & 4 ? q.x : q.y;
        float one = own + __shfl_xor_sync(0xffffffffu, other, 4);
#pragma unroll
        for (int o = P; o < 4; o <<= 1) one += __shfl_xor_sync(0xffffffffu, one, o);
        red[warp][piece * 8 + (lane >> 4) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1)] = one;
        __syncthreads();
        if (threadIdx.x < TT) {
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < kLnWideThreads / 32; ++w) t += red[w][lane];
            sums[lane] = t;
        }
        __syncthreads();
        const float4 lo = *reinterpret_cast<const float4*>(&sums[piece * 8]), hi = *reinterpret_cast<const float4*>(&sums[piece * 8 + 4]);
        f[0] = pair_of(lo.x, lo.y); f[1] = pair_of(lo.z, lo.w); f[2] = pair_of(hi.x, hi.y); f[3] = pair_of(hi.z, hi.w);
    };
    const int last = in ? (hidden - r0 + kRows - 1) / kRows : 0;               // pieces of this thread
    const int64_t at0 = (int64_t)r0 * tokens + t0, turn = (int64_t)kRows * tokens;
    uint4 v[NV];
    // The passes unpack v anew: without this the compiler keeps 8 * NV floats from one to the next, and spills.
    auto forget = [&]() {
#pragma unroll
        for (int j = 0; j < NV; ++j) asm volatile("" : "+r"(v[j].x), "+r"(v[j].y), "+r"(v[j].z), "+r"(v[j].w));
    };
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = j < last ? __ldg(reinterpret_cast<const uint4*>(x + at0 + j * turn)) : make_uint4(0, 0, 0, 0);
    if (bias)
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (j < last) {
                f32x2 f[4];
                unpack4(v[j], f);
                const float b = __half2float(__ldg(bias + r0 + j * kRows));
#pragma unroll
                for (int e = 0; e < 4; ++e) f[e] = add2(f[e], pair_of(b, b));
                v[j] = pack4(f);
            }
    if (add)
#pragma unroll
        for (int j0 = 0; j0 < NV; j0 += kPair) {
            uint4 a[kPair];
#pragma unroll
            for (int q = 0; q < kPair; ++q) a[q] = j0 + q < last ? __ldg(reinterpret_cast<const uint4*>(add + at0 + (j0 + q) * turn)) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int q = 0; q < kPair; ++q) {
                f32x2 f[4], g[4];
                unpack4(v[j0 + q], f);
                unpack4(a[q], g);
#pragma unroll
                for (int e = 0; e < 4; ++e) f[e] = add2(f[e], g[e]);
                v[j0 + q] = pack4(f);
                if (j0 + q < last) *reinterpret_cast<uint4*>(sum_out + at0 + (j0 + q) * turn) = v[j0 + q];
            }
        }
    forget();
    f32x2 mean[4] = {0, 0, 0, 0}, var[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        f32x2 f[4];
        unpack4(v[j], f);
#pragma unroll
        for (int e = 0; e < 4; ++e) mean[e] = add2(mean[e], f[e]);                 // (pieces past the last are zeros)
    }
    total(mean, whole[0]);
    forget();
    const float inv = 1.f / (float)hidden;
#pragma unroll
    for (int e = 0; e < 4; ++e) mean[e] = mul2(mean[e], pair_of(-inv, -inv));      // its negative
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (j < last) {
            f32x2 f[4];
            unpack4(v[j], f);
#pragma unroll
            for (int e = 0; e < 4; ++e) { const f32x2 d = add2(f[e], mean[e]); var[e] = fma2(d, d, var[e]); }
        }
    total(var, whole[1]);
    forget();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 s = floats_of(var[e]);
        var[e] = pair_of(rsqrtf(fmaf(s.x, inv, eps)), rsqrtf(fmaf(s.y, inv, eps)));
    }
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (j < last) {
            f32x2 f[4];
            unpack4(v[j], f);
            const float g = __half2float(__ldg(gamma + r0 + j * kRows)), b = __half2float(__ldg(beta + r0 + j * kRows));
#pragma unroll
            for (int e = 0; e < 4; ++e) f[e] = fma2(mul2(add2(f[e], mean[e]), var[e]), pair_of(g, g), pair_of(b, b));
            *reinterpret_cast<uint4*>(out + at0 + j * turn) = pack4(f);
        }
}

template <int TT, int NV>
__global__ void __launch_bounds__(kLnWideThreads, 2)
layer_norm_fm_regs_kernel(int hidden, int tokens, const __half* __restrict__ x, const __half* __restrict__ bias, const __half* __restrict__ add,
                          __half* __restrict__ sum_out, const __half* __restrict__ gamma, const __half* __restrict__ beta, float eps,
                          __half* __restrict__ out) {
    layer_norm_tile<TT, NV>(blockIdx.x, hidden, tokens, x, bias, add, sum_out, gamma, beta, eps, out);
}

// The first CTAs write the dense copies of a layer's operands, the others normalise its input: neither needs the other, the copies are chains
// of look-ups and the input is traffic.  768 wide, 32 x 512 tokens: 14.0 and 12.4 us one after the other and a launch between, 23.6 together; the
// layer takes 335 us where it takes 339, with 4 x 512 tokens 104.8 (107.2), 16 x 512 213.2 (216.9).
template <int TT, int NV>
__global__ void __launch_bounds__(kLnWideThreads, 2)
layer_norm_copies_kernel(const __grid_constant__ ExpandSet s, int hidden, int tokens, const __half* __restrict__ x, const __half* __restrict__ gamma,
                         const __half* __restrict__ beta, float eps, __half* __restrict__ out) {
    __shared__ int slot[kExpandChunk];
    const int copies = s.first[s.count];
    if ((int)blockIdx.x < copies) expand_of_set(s, blockIdx.x, slot);
    else layer_norm_tile<TT, NV>(blockIdx.x - copies, hidden, tokens, x, nullptr, nullptr, nullptr, gamma, beta, eps, out);
}

// Calls f with tokens per tile and pieces per thread of the kernels above; false: a tile goes through shared memory.
template <typename F>
bool with_tile(int hidden, int tokens, int sms, F&& f) {
    using std::integral_constant;
    auto go = [&](auto tt, auto nv) { f(tt, nv); return true; };
    constexpr integral_constant<int, 1> k1{};
    constexpr integral_constant<int, 2> k2{};
    constexpr integral_constant<int, 4> k4{};
    constexpr integral_constant<int, 6> k6{};
    constexpr integral_constant<int, 8> k8{};
    constexpr integral_constant<int, 16> k16{};
    constexpr integral_constant<int, 32> k32{};
    // as many tokens per CTA as give every SM one
    if (tokens >= 32 * sms) {
        if (hidden > 1024) return false;
        return hidden <= 256 ? go(k32, k2) : hidden <= 512 ? go(k32, k4) : hidden <= 768 ? go(k32, k6) : go(k32, k8);
    }
    if (tokens >= 16 * sms && hidden <= 1024) return hidden <= 256 ? go(k16, k1) : hidden <= 512 ? go(k16, k2) : go(k16, k4);
    return hidden <= 512 ? go(k8, k1) : hidden <= 1024 ? go(k8, k2) : go(k8, k6);
}

// out = x + bias + add, rounded after each addition; one 16-byte piece per thread.
__global__ void __launch_bounds__(256)
add_bias_fm_kernel(int rows, int tokens, const __half* __restrict__ x, const __half* __restrict__ bias, const __half* __restrict__ add,
                   __half* __restrict__ out) {
    const int64_t pieces = (int64_t)rows * (tokens / 8);
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < pieces; i += (int64_t)gridDim.x * 256) {
        float f[8], g[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(x) + i), f);
        unpack8(__ldg(reinterpret_cast<const uint4*>(add) + i), g);
        const float b = __half2float(__ldg(bias + i / (tokens / 8)));
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __half2float(__float2half_rn(f[e] + b)) + g[e];
        reinterpret_cast<uint4*>(out)[i] = pack8(f);
    }
}

// ---- attention ------------------------------------------------------------------------------------
// One CTA: 64 queries of one head of one sequence, four warps of 16 queries; keys and values pass through shared memory 64
// tokens at a time (two buffers, cp.async), the running maximum, sum and output of a query stay in registers.  Head width
// 64.  Everything is read as it lies, [feature][token]: q and k are fetched by transposing ldmatrix, v by the plain one.
// Probabilities are two fp16 numbers, p = hi + lo, and two matrix instructions: 22 bits of it, or 2^-35 of the query's largest
// probability where that is more.  The score path needs no such split, its operands are fp16 already.  The matrix unit truncates
// when it adds, so the sums over a block of 64 keys start from zero and join the others by an addition that rounds to nearest.
// Optional biases of q and v (per feature) are added here: q's to the fragments, v's to the result, since the probabilities
// of a query sum to one; one of k would add the same number to all scores of a query, which the softmax does not see.
// Bound by the matrix instructions (96 of m16n8k16 per warp and 64 keys) and the exponentials.  12 heads, 32 x 512 tokens:
// 140 us (136 with one running sum), 1350 us as torch's unfused fp32 path (the strided views rule out its fused kernels).
// Distance from 64 bits there, of which rounding the result is 2.075240e-4: 2.075243e-4 (one running sum 2.075284e-4, torch
// 2.075246e-4), and no larger than torch's from 64 to 512 tokens, scores of size 0.01 to 100.
constexpr int kHd = 64, kTile = 64, kAttnThreads = 128;
constexpr int kTileBytes = kHd * kTile * 2;                 // 8 KB: [64 features][64 tokens], pieces swizzled by the feature

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
    const uint32_t bytes = valid ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// address of the 16-byte piece (feature row, piece) of a tile
__device__ __forceinline__ uint32_t at(uint32_t tile, int row, int piece) { return tile + row * 128 + ((piece ^ (row & 7)) << 4); }

// Which elements of two fp16 numbers are infinite or NaN, as a mask of their bits.
__device__ __forceinline__ uint32_t nonfinite(uint32_t x) {
    return ((x & 0x7c00u) == 0x7c00u ? 0xffffu : 0u) | ((x & 0x7c000000u) == 0x7c000000u ? 0xffff0000u : 0u);
}

// Sums over all keys for the 16 queries of a warp: o[block of 8 features][query g: 0, 1; g + 8: 2, 3], and 1 / sum of
// probabilities.  The whole CTA takes part.
// SPECIAL: infinities and NaNs of v are multiplied by whether a probability is zero and not by its two terms, of which the
// low one may be zero or negative (which would make NaN of an infinite result).
template <bool SPECIAL>
__device__ __forceinline__ void attend(int seq, int64_t tokens, int64_t base, int q0, const __half* __restrict__ q, const __half* __restrict__ k,
                                       const __half* __restrict__ v, const __half* __restrict__ bias_q, uint32_t s_q, float (&o)[8][4],
                                       float (&inv)[2]) {
    const uint32_t s_kv = s_q + kTileBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3;
    auto load = [&](uint32_t dst, const __half* src, int s0) {
        for (int x = threadIdx.x; x < kHd * 8; x += kAttnThreads) {
            const int row = x >> 3, piece = x & 7, s = s0 + piece * 8;
            const bool ok = s < seq;                                // seq % 8 == 0: a piece is all in or all out
            cp16(at(dst, row, piece), src + base + (int64_t)row * tokens + (ok ? s : 0), ok);
        }
    };
    load(s_q, q, q0);
    load(s_kv, k, 0);
    load(s_kv + kTileBytes, v, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");

    constexpr float kScale = 0.125f * 1.44269504088896340736f;      // 1 / sqrt(64), in powers of two
    constexpr float kLift = 10.f;                                   // probabilities are carried times 2^10: low halves are normal numbers down to 2^-13 of the largest one
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
    uint32_t qf[4][4];                                              // [16 features][fragment]
    const int rounds = (seq + kTile - 1) / kTile;
    for (int it = 0; it < rounds; ++it) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        named_barrier_sync(1, kAttnThreads);                        // this round's tiles are in, the other buffer is free
        if (it + 1 < rounds) {
            const uint32_t next = s_kv + ((it + 1) & 1) * 2 * kTileBytes;
            load(next, k, (it + 1) * kTile);
            load(next + kTileBytes, v, (it + 1) * kTile);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const uint32_t s_k = s_kv + (it & 1) * 2 * kTileBytes, s_v = s_k + kTileBytes;
        if (it == 0) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)                          // matrices (features lo, tokens lo), (lo, hi), (hi, lo), (hi, hi)
                ldsm4_t(qf[kk], at(s_q, kk * 16 + (lane >> 4) * 8 + (lane & 7), warp * 2 + ((lane >> 3) & 1)));
            if (bias_q) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int f = 0; f < 4; ++f) {                   // features 2t, 2t + 1 of the fragment's half
                        const __half* b = bias_q + kk * 16 + (f >> 1) * 8 + 2 * t;
                        const __half2 s2 = __hadd2(*reinterpret_cast<const __half2*>(&qf[kk][f]), __halves2half2(b[0], b[1]));
                        qf[kk][f] = *reinterpret_cast<const uint32_t*>(&s2);
                    }
            }
        }
        float s[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) {                        // two blocks of eight keys
                uint32_t b[4];                                      // (features lo, keys a), (hi, a), (lo, b), (hi, b)
                ldsm4_t(b, at(s_k, kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), n2 * 2 + (lane >> 4)));
                mma(s[2 * n2], qf[kk], b[0], b[1]);
                mma(s[2 * n2 + 1], qf[kk], b[2], b[3]);
            }
        const int left = seq - it * kTile;
        if (left < kTile) {
#pragma unroll
            for (int n = 0; n < 8; ++n)
                if (n * 8 >= left)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[n][e] = -INFINITY;
        }
        // rows g (elements 0, 1) and g + 8 (2, 3) of the warp's 16 queries
        float shift[2], keep[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float mx = m[h];
#pragma unroll
            for (int n = 0; n < 8; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * h], s[n][2 * h + 1]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            keep[h] = mx == -INFINITY ? 1.f : exp2f((m[h] - mx) * kScale);
            m[h] = mx;
            shift[h] = mx == -INFINITY ? 0.f : mx;
            l[h] *= keep[h];
        }
        uint32_t hi[4][4], lo[4][4], nonzero = 0;                   // [16 keys][fragment]; a bit per probability
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)                              // score blocks 2 kk and 2 kk + 1 are the fragment
#pragma unroll
            for (int f = 0; f < 4; ++f) {                           // (queries lo, keys lo), (hi, lo), (lo, hi), (hi, hi)
                const int n = 2 * kk + (f >> 1), h = f & 1;
                const float p0 = exp2f(fmaf(s[n][2 * h] - shift[h], kScale, kLift)), p1 = exp2f(fmaf(s[n][2 * h + 1] - shift[h], kScale, kLift));
                l[h] += p0 + p1;
                const __half2 ph = __floats2half2_rn(p0, p1);
                const float2 back = __half22float2(ph);
                const __half2 pl = __floats2half2_rn(p0 - back.x, p1 - back.y);
                hi[kk][f] = *reinterpret_cast<const uint32_t*>(&ph);
                lo[kk][f] = *reinterpret_cast<const uint32_t*>(&pl);
                if constexpr (SPECIAL) nonzero |= (p0 > 0.f ? 1u : 0u) << (8 * kk + 2 * f) | (p1 > 0.f ? 2u : 0u) << (8 * kk + 2 * f);
            }
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {                            // two blocks of eight output features
            float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint32_t b[4];                                      // (features a, keys lo), (a, hi), (b, lo), (b, hi)
                ldsm4(b, at(s_v, n2 * 16 + (lane >> 4) * 8 + (lane & 7), kk * 2 + ((lane >> 3) & 1)));
                if constexpr (SPECIAL) {
                    uint32_t x[4], some[4];
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        x[f] = b[f] & nonfinite(b[f]);
                        b[f] ^= x[f];
                        some[f] = (nonzero >> (8 * kk + 2 * f) & 1u) * 0x3c00u | (nonzero >> (8 * kk + 2 * f + 1) & 1u) * 0x3c000000u;
                    }
                    mma(d[0], some, x[0], x[1]);
                    mma(d[1], some, x[2], x[3]);
                }
                mma(d[0], lo[kk], b[0], b[1]);
                mma(d[1], lo[kk], b[2], b[3]);
                mma(d[0], hi[kk], b[0], b[1]);
                mma(d[1], hi[kk], b[2], b[3]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[2 * n2 + j][e] = fmaf(o[2 * n2 + j][e], keep[e >> 1], d[j][e]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
        inv[h] = 1.f / l[h];                                       // no score above -inf: 0 * inf, NaN
    }
}

// The warp's 16 columns of the output tile [feature][query] take the place of its queries, and go out.
__device__ __forceinline__ void store_queries(int seq, int64_t tokens, int64_t base, int q0, int head, const __half* __restrict__ bias_v,
                                              uint8_t* smem, const float (&o)[8][4], const float (&inv)[2], __half* __restrict__ out) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    __half* tile = reinterpret_cast<__half*>(smem);
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = n * 8 + 2 * t + (e & 1), piece = warp * 2 + (e >> 1);
            const float b = bias_v ? __half2float(bias_v[head * kHd + row]) : 0.f;
            tile[row * 64 + ((piece ^ (row & 7)) << 3) + g] = __float2half_rn(fmaf(o[n][e], inv[e >> 1], b));
        }
    __syncwarp();
#pragma unroll
    for (int x = lane; x < kHd * 2; x += 32) {
        const int row = x >> 1, piece = warp * 2 + (x & 1), s = q0 + piece * 8;
        if (s < seq)
            *reinterpret_cast<uint4*>(out + base + (int64_t)row * tokens + s) = *reinterpret_cast<const uint4*>(tile + row * 64 + ((piece ^ (row & 7)) << 3));
    }
}

__global__ void __launch_bounds__(kAttnThreads, 4)
attention_fm_kernel(int seq, int64_t tokens, const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v,
                    const __half* __restrict__ bias_q, const __half* __restrict__ bias_v, __half* __restrict__ out) {
    __shared__ __align__(128) uint8_t smem[5 * kTileBytes];         // q (later the output), two buffers of k and v
    const int q0 = blockIdx.x * kTile, head = blockIdx.y;
    const int64_t base = (int64_t)head * kHd * tokens + (int64_t)blockIdx.z * seq;
    if (bias_q) bias_q += head * kHd;
    float o[8][4], inv[2];
    attend<false>(seq, tokens, base, q0, q, k, v, bias_q, smem_u32(smem), o, inv);
    bool nan = false;
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) nan |= isnan(o[n][e]);
    // something infinite or NaN went in (the barrier also frees the buffers)
    if (__syncthreads_or(nan)) attend<true>(seq, tokens, base, q0, q, k, v, bias_q, smem_u32(smem), o, inv);
    store_queries(seq, tokens, base, q0, head, bias_v, smem, o, inv, out);
}

// ---- attention on tcgen05 ---------------------------------------------------------------------------
// One CTA: 128 queries of one head of one sequence.  Four warps hold a query per thread: they read its 64 scores of a block of keys
// from tensor memory, keep the running maximum, sum and output in registers and put the probabilities (two fp16 numbers
// each) back in place of the scores; a fifth warp requests tiles by TMA and issues the products.  Keys and values pass through
// three stages of 64 tokens; scores and partial outputs have two buffers each in tensor memory, so the scores of the
// next block are computed while this block's probabilities are, and a partial output is taken one block later.
// The arithmetic is attend's: blocks of 64 keys, sums of a block from zero, joined in round-to-nearest.
// Bound by the softmax warps: about seven instructions per score (additions, products and the joining of outputs work on pairs of
// numbers, each rounded as by itself; one number at a time it was ten), and the waits between them and the products, which two CTAs per SM
// do not fill.  12 heads, 32 x 512 tokens: 71 us, 78 one number at a time (attention_fm_kernel 141; 85 with the first requests after the
// set-up); one number at a time 16 x 512 40 (75), 1 x 2048 44 (83).  Distance from 64 bits as there: 2.074969e-4 against 2.074970e-4 (scores of size 1), 2.073688e-4 against 2.073688e-4
// (size 5).  A CTA that walks over tiles with the next one's operands on their way takes 96 us.
constexpr int kTcQueries = 128, kTcStages = 3, kTcThreads = 160;
struct TcSmem {
    static constexpr int kQ = 0;                                     // two chunks of [64 features][64 queries]
    static constexpr int kKv = 2 * kTileBytes;                       // [stage][k, v][64 features][64 keys]
    static constexpr int kBar = kKv + kTcStages * 2 * kTileBytes;
    static constexpr int kBars = kTcStages + 1 + 8;
    static constexpr int kTmem = kBar + kBars * 8;
    static constexpr int kAbort = kTmem + 8;
    static constexpr int kBytes = kAbort + 8;
    static constexpr int kDynamic = kBytes + 1024;
    static_assert(5 * kTileBytes <= kBar, "attend's tiles fit in place of the stages");
};
constexpr uint32_t kTcTmemCols = 256;                                // scores / probabilities 2 x 64, partial outputs 2 x 64

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__global__ void __launch_bounds__(kTcThreads, 2)
attention_tc_kernel(int seq, int64_t tokens, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const __half* __restrict__ q, const __half* __restrict__ k,
                    const __half* __restrict__ v, const __half* __restrict__ bias_q, const __half* __restrict__ bias_v,
                    __half* __restrict__ out) {
    using L = TcSmem;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar_kv_full = sbase + L::kBar, bar_q = bar_kv_full + 8 * kTcStages;
    const uint32_t bar_s_full = bar_q + 8, bar_p_full = bar_s_full + 16, bar_o_full = bar_p_full + 16, bar_o_free = bar_o_full + 16;
    volatile uint32_t* tmem_at = reinterpret_cast<volatile uint32_t*>(smem + L::kTmem);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kAbort);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q0 = blockIdx.x * kTcQueries, head = blockIdx.y, b = blockIdx.z;
    const int rounds = (seq + kTile - 1) / kTile;
    auto tile = [&](int stage, int which) { return sbase + L::kKv + (stage * 2 + which) * kTileBytes; };
    int loaded = 0;
    auto request = [&]() {                                           // the next block's tiles; their stage is free
        const int s = loaded % kTcStages;
        mbar_arrive_expect_tx(bar_kv_full + 8 * s, 2 * kTileBytes);
        tma_load_3d(tile(s, 0), &tmap_k, loaded * kTile, head * kHd, b, bar_kv_full + 8 * s);
        tma_load_3d(tile(s, 1), &tmap_v, loaded * kTile, head * kHd, b, bar_kv_full + 8 * s);
        ++loaded;
    };

    if (warp == 4) {
        if (lane == 0) {
            for (int s = 0; s < kTcStages; ++s) mbar_init(bar_kv_full + 8 * s, 1);
            mbar_init(bar_q, 1);
            for (int i = 0; i < 2; ++i) {
                mbar_init(bar_s_full + 8 * i, 1);
                mbar_init(bar_p_full + 8 * i, 4);
                mbar_init(bar_o_full + 8 * i, 1);
                mbar_init(bar_o_free + 8 * i, 4);
            }
            *abort_flag = 0;
            mbar_fence_init();
            // on their way while the others start
            mbar_arrive_expect_tx(bar_q, 2 * kTileBytes);
            tma_load_3d(sbase + L::kQ, &tmap_q, q0, head * kHd, b, bar_q);
            tma_load_3d(sbase + L::kQ + kTileBytes, &tmap_q, q0 + 64, head * kHd, b, bar_q);
            while (loaded < min(rounds, kTcStages)) request();
        }
        __syncwarp();
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_at)), kTcTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_at;

    bool nan = false, done = false;
    f32x2 o[kHd / 2], l[2] = {0, 0};                                // of the softmax warps, in pairs
    if (warp == 4) {
        if (lane == 0) {
            // queries are in when the softmax warps say so (they add the bias first): their arrival is the first phase of o_free[0]
            bool ok = mbar_wait(bar_o_free, 0, abort_flag, kStatusWaitAttention);
            constexpr uint32_t idesc_s = make_idesc_f16_f32(kTcQueries, kTile, true, true);
            constexpr uint32_t idesc_o = make_idesc_f16_f32(kTcQueries, kHd, false, false);
            auto scores = [&](int it) -> bool {
                const int s = it % kTcStages;
                if (!mbar_wait(bar_kv_full + 8 * s, (it / kTcStages) & 1, abort_flag, kStatusWaitAttention)) return false;
                tc_fence_after_sync();
                for (int kk = 0; kk < 4; ++kk)
                    tc_mma_f16(tmem + (it & 1) * kTile, make_smem_desc(sbase + L::kQ + kk * 2048, kTileBytes, 1024, 2),
                               make_smem_desc(tile(s, 0) + kk * 2048, kTileBytes, 1024, 2), idesc_s, kk > 0 ? 1u : 0u);
                tc_commit(bar_s_full + 8 * (it & 1));
                return true;
            };
            ok = ok && scores(0);
            for (int it = 0; ok && it < rounds; ++it) {
                const int buf = it & 1, s = it % kTcStages;
                if (it > 0) {
                    // the block before is done: its stage is free, and so is the buffer that the next scores go to
                    if (!mbar_wait(bar_o_full + 8 * (buf ^ 1), ((it - 1) >> 1) & 1, abort_flag, kStatusWaitAttention)) break;
                    tc_fence_after_sync();
                    if (loaded < rounds) request();
                }
                if (it + 1 < rounds && !scores(it + 1)) break;
                if (!mbar_wait(bar_p_full + 8 * buf, (it >> 1) & 1, abort_flag, kStatusWaitAttention)) break;
                // the partial output two blocks ago has been taken (buffer 0 is one phase ahead, see above)
                if (it >= 2 && !mbar_wait(bar_o_free + 8 * buf, (((it - 2) >> 1) + (buf == 0 ? 1 : 0)) & 1, abort_flag, kStatusWaitAttention)) break;
                tc_fence_after_sync();
                const uint32_t p = tmem + buf * kTile, o = tmem + 2 * kTile + buf * kHd;
                for (int part = 0; part < 2; ++part)                // low halves first
                    for (int kk = 0; kk < 4; ++kk)
                        tc_mma_f16_ts(o, p + (part == 0 ? 32 : 0) + kk * 8, make_smem_desc(tile(s, 1) + kk * 32, 16, 1024, 2), idesc_o,
                                      part + kk > 0 ? 1u : 0u);
                tc_commit(bar_o_full + 8 * buf);
            }
        }
    } else {
        const int row = threadIdx.x;                                // query of the tile
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        constexpr float kScale = 0.125f * 1.44269504088896340736f;
        constexpr float kLift = 10.f;
        bool ok = mbar_wait(bar_q, 0, abort_flag, kStatusWaitAttention);
        if (ok && bias_q) {
            for (int x = threadIdx.x; x < kHd * 16; x += 128) {     // 64 features x 16 pieces of eight queries
                const int f = x >> 4, piece = x & 15;
                uint4* at16 = reinterpret_cast<uint4*>(smem + L::kQ + (piece >> 3) * kTileBytes + f * 128 + (((piece & 7) ^ (f & 7)) << 4));
                uint4 w = *at16;
                const __half2 bb = __half2half2(bias_q[head * kHd + f]);
                uint32_t* h = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const __half2 sum = __hadd2(*reinterpret_cast<const __half2*>(&h[e]), bb);
                    h[e] = *reinterpret_cast<const uint32_t*>(&sum);
                }
                *at16 = w;
            }
            fence_proxy_async_smem();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_o_free);
        float m = -INFINITY, keep = 1.f;
#pragma unroll
        for (int f = 0; f < kHd / 2; ++f) o[f] = 0;
        // adds the partial output of block it: o = o * factor + partial
        auto join = [&](int it, float factor) -> bool {
            const int buf = it & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(bar_o_full + 8 * buf, (it >> 1) & 1, abort_flag, kStatusWaitAttention))) return false;
            tc_fence_after_sync();
            const f32x2 both = pair_of(factor, factor);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t d[32];
                tmem_ld_x32(tmem + lanes + 2 * kTile + buf * kHd + h * 32, d);
                tc_wait_ld();
#pragma unroll
                for (int f = 0; f < 16; ++f)
                    o[h * 16 + f] = fma2(o[h * 16 + f], both, pair_of(__uint_as_float(d[2 * f]), __uint_as_float(d[2 * f + 1])));
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_o_free + 8 * buf);
            return true;
        };
        for (int it = 0; it < rounds; ++it) {
            const int buf = it & 1;
            if (!__all_sync(0xffffffffu, ok && mbar_wait(bar_s_full + 8 * buf, (it >> 1) & 1, abort_flag, kStatusWaitAttention))) { ok = false; break; }
            tc_fence_after_sync();
            uint32_t s[2][32];
            tmem_ld_x32(tmem + lanes + buf * kTile, s[0]);
            tmem_ld_x32(tmem + lanes + buf * kTile + 32, s[1]);
            tc_wait_ld();
            const int left = seq - it * kTile;
            if (left < kTile) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int n = 0; n < 32; ++n)
                        if (h * 32 + n >= left) s[h][n] = 0xff800000u;       // -inf
            }
            float mx[4] = {m, m, m, m};
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int n = 0; n < 32; ++n) mx[n & 3] = fmaxf(mx[n & 3], __uint_as_float(s[h][n]));
            mx[0] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const float last = keep;
            keep = mx[0] == -INFINITY ? 1.f : exp2f((m - mx[0]) * kScale);
            m = mx[0];
            const float shift = m == -INFINITY ? 0.f : m;
#pragma unroll
            for (int e = 0; e < 2; ++e) l[e] = mul2(l[e], pair_of(keep, keep));
            const f32x2 less = pair_of(-shift, -shift), scale = pair_of(kScale, kScale), lift = pair_of(kLift, kLift);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    const uint32_t* const at2 = &s[h >> 1][(h & 1) * 16 + 2 * n];
                    const float2 x = floats_of(fma2(add2(pair_of(__uint_as_float(at2[0]), __uint_as_float(at2[1])), less), scale, lift));
                    const float p0 = ex2(x.x), p1 = ex2(x.y);
                    const f32x2 p = pair_of(p0, p1);
                    l[n & 1] = add2(l[n & 1], p);
                    const __half2 ph = __floats2half2_rn(p0, p1);
                    const float2 back = __half22float2(ph);
                    const float2 rest = floats_of(add2(p, pair_of(-back.x, -back.y)));
                    const __half2 pl = __floats2half2_rn(rest.x, rest.y);
                    hi[n] = *reinterpret_cast<const uint32_t*>(&ph);
                    lo[n] = *reinterpret_cast<const uint32_t*>(&pl);
                }
                tmem_st_x8(tmem + lanes + buf * kTile + h * 8, hi);
                tmem_st_x8(tmem + lanes + buf * kTile + 32 + h * 8, lo);
            }
            tc_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_full + 8 * buf);
            if (it > 0 && !join(it - 1, last)) { ok = false; break; }
        }
        done = ok && join(rounds - 1, keep) && q0 + row < seq;
        if (done)
#pragma unroll
            for (int f = 0; f < kHd / 2; ++f) { const float2 x = floats_of(o[f]); nan |= isnan(x.x) || isnan(x.y); }
    }
    tc_fence_before_sync();
    nan = __syncthreads_or(nan);
    if (warp == 4) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTcTmemCols);
    }
    if (done && !nan) {                                             // (out may be q, which a second pass reads again)
        const float2 l01 = floats_of(l[0]), l23 = floats_of(l[1]);
        const float inv = 1.f / ((l01.x + l01.y) + (l23.x + l23.y));
        __half* dst = out + (int64_t)head * kHd * tokens + (int64_t)b * seq + q0 + threadIdx.x;
#pragma unroll
        for (int f = 0; f < kHd; ++f) {
            const float2 x = floats_of(o[f >> 1]);
            dst[f * tokens] = __float2half_rn(fmaf(f & 1 ? x.y : x.x, inv, bias_v ? __half2float(bias_v[head * kHd + f]) : 0.f));
        }
    }
    // something infinite or NaN went in: again, with infinities and NaNs of v apart, 64 queries at a time
    if (nan && warp < 4) {
        const int64_t base = (int64_t)head * kHd * tokens + (int64_t)b * seq;
        for (int at = q0; at < min(seq, q0 + kTcQueries); at += kTile) {
            float o[8][4], inv[2];
            attend<true>(seq, tokens, base, at, q, k, v, bias_q ? bias_q + head * kHd : nullptr, sbase, o, inv);
            store_queries(seq, tokens, base, at, head, bias_v, smem, o, inv, out);
            named_barrier_sync(1, kAttnThreads);
        }
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
    static EncodeFn cached = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<EncodeFn>(fn);
    }();
    return cached;
}
// {token of a sequence, feature, sequence}, boxes of 64 tokens x 64 features; tokens past a sequence read as zeros
bool encode_tokens(EncodeFn enc, CUtensorMap* m, const void* x, int hidden, int batch, int seq) {
    const cuuint64_t dim[3] = {(cuuint64_t)seq, (cuuint64_t)hidden, (cuuint64_t)batch};
    const cuuint64_t stride[2] = {(cuuint64_t)batch * seq * 2, (cuuint64_t)seq * 2};
    const cuuint32_t box[3] = {kTile, kHd, 1}, step[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), dim, stride, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool piece_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }   // null passes

}  // namespace enc
}  // namespace sspmm_b200

using namespace sspmm_b200;

extern "C" {

int sspmm_layer_norm_fm(int hidden, int tokens, const void* x, const void* bias, const void* add, void* sum_out, const void* gamma, const void* beta,
                        float eps, void* out, void* stream) {
    set_error("%s", "");
    if (hidden <= 0 || hidden > 3072 || tokens < 0 || tokens % 8 != 0 || !x || !gamma || !beta || !out || (add && !sum_out) ||
        !enc::piece_aligned(x) || !enc::piece_aligned(add) || !enc::piece_aligned(sum_out) || !enc::piece_aligned(out)) {
        set_error("LayerNorm: bad argument (hidden=%d tokens=%d)", hidden, tokens);
        return (int)cudaErrorInvalidValue;
    }
    if (tokens == 0) return 0;
    const int sms = current_device_sm_count();
    if (sms <= 0) return (int)cudaErrorNoDevice;
    const __half *hx = static_cast<const __half*>(x), *hb = static_cast<const __half*>(bias), *ha = static_cast<const __half*>(add);
    const __half *hg = static_cast<const __half*>(gamma), *ht = static_cast<const __half*>(beta);
    __half *hs = static_cast<__half*>(sum_out), *ho = static_cast<__half*>(out);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool done = enc::with_tile(hidden, tokens, sms, [&](auto tt, auto nv) {
        enc::layer_norm_fm_regs_kernel<tt, nv><<<(tokens + tt - 1) / tt, enc::kLnWideThreads, 0, st>>>(hidden, tokens, hx, hb, ha, hs, hg, ht, eps, ho);
    });
    if (!done) {
        static DeviceOnce once;
        if (!once.done()) {
            const cudaError_t e = cudaFuncSetAttribute(enc::layer_norm_fm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 3072 * 32 * 2);
            if (e != cudaSuccess) { set_error("LayerNorm: %s", cudaGetErrorString(e)); return (int)e; }
            once.mark();
        }
        enc::layer_norm_fm_kernel<<<(tokens + 31) / 32, enc::kLnThreads, (size_t)hidden * 32 * 2, st>>>(hidden, tokens, hx, hb, ha, hs, hg, ht, eps, ho);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("LayerNorm launch: %s", cudaGetErrorString(e)); return (int)e; }
    return 0;
}

int sspmm_layer_norm_copies(int count, const sspmm_dense_operand* operands, int N, void* room, int hidden, int tokens, const void* x, const void* gamma,
                            const void* beta, float eps, void* out, void* stream) {
    set_error("%s", "");
    if (hidden <= 0 || hidden > 3072 || tokens <= 0 || tokens % 8 != 0 || !x || !gamma || !beta || !out || !room || !enc::piece_aligned(x) ||
        !enc::piece_aligned(out)) {
        set_error("LayerNorm with copies: bad argument (hidden=%d tokens=%d)", hidden, tokens);
        return (int)cudaErrorInvalidValue;
    }
    SpmmArgs a[kMaxCopies];
    __half* at[kMaxCopies];
    int copies = 0;
    int64_t offsets[kMaxCopies], bytes = 0;
    const int rc = collect_copies(count, operands, N, room, a, at, &copies, offsets, &bytes);
    if (rc != 0) return rc;
    const int sms = current_device_sm_count();
    if (sms <= 0) return (int)cudaErrorNoDevice;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ExpandSet s;
    cudaError_t e = make_expand_set(a, at, copies, sms, &s);
    if (e != cudaSuccess) { set_error("dense copies: %s", cudaGetErrorString(e)); return (int)e; }
    const __half *hx = static_cast<const __half*>(x), *hg = static_cast<const __half*>(gamma), *hb = static_cast<const __half*>(beta);
    if (enc::with_tile(hidden, tokens, sms, [&](auto tt, auto nv) {
            enc::layer_norm_copies_kernel<tt, nv><<<s.first[s.count] + (tokens + tt - 1) / tt, enc::kLnWideThreads, 0, st>>>(
                s, hidden, tokens, hx, hg, hb, eps, static_cast<__half*>(out));
        })) {
        e = cudaGetLastError();
        if (e != cudaSuccess) { set_error("LayerNorm launch: %s", cudaGetErrorString(e)); return (int)e; }
        return 0;
    }
    e = launch_expand_set(a, at, copies, st);
    if (e != cudaSuccess) { set_error("dense copies: %s", cudaGetErrorString(e)); return (int)e; }
    return sspmm_layer_norm_fm(hidden, tokens, x, nullptr, nullptr, nullptr, gamma, beta, eps, out, stream);
}

int sspmm_add_bias_fm(int rows, int tokens, const void* x, const void* bias, const void* add, void* out, void* stream) {
    set_error("%s", "");
    if (rows < 0 || tokens < 0 || tokens % 8 != 0 || !x || !bias || !add || !out || !enc::piece_aligned(x) || !enc::piece_aligned(add) ||
        !enc::piece_aligned(out)) {
        set_error("bias and residual: bad argument (rows=%d tokens=%d)", rows, tokens);
        return (int)cudaErrorInvalidValue;
    }
    const int64_t pieces = (int64_t)rows * (tokens / 8);
    if (pieces == 0) return 0;
    const int sms = current_device_sm_count();
    if (sms <= 0) return (int)cudaErrorNoDevice;
    const int64_t blocks = (pieces + 255) / 256, most = (int64_t)sms * 16;
    enc::add_bias_fm_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        rows, tokens, static_cast<const __half*>(x), static_cast<const __half*>(bias), static_cast<const __half*>(add), static_cast<__half*>(out));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("bias and residual launch: %s", cudaGetErrorString(e)); return (int)e; }
    return 0;
}

int sspmm_attention_fm(int heads, int head_dim, int batch, int seq, const void* q, const void* k, const void* v, const void* bias_q,
                       const void* bias_v, void* out, void* stream) {
    return sspmm_attention_fm_as(0, heads, head_dim, batch, seq, q, k, v, bias_q, bias_v, out, stream, nullptr);
}

int sspmm_attention_fm_as(int kernel, int heads, int head_dim, int batch, int seq, const void* q, const void* k, const void* v,
                          const void* bias_q, const void* bias_v, void* out, void* stream, int* taken) {
    set_error("%s", "");
    if (taken) *taken = 0;
    if (kernel < 0 || kernel > 2) { set_error("attention kernel must be 0, 1 or 2"); return (int)cudaErrorInvalidValue; }
    if (heads < 0 || batch < 0 || seq < 0 || head_dim != enc::kHd || seq % 8 != 0 || heads > 65535 || batch > 65535 || !q || !k || !v || !out ||
        !enc::piece_aligned(q) || !enc::piece_aligned(k) || !enc::piece_aligned(v) || !enc::piece_aligned(out)) {
        set_error("attention: bad argument (heads=%d head_dim=%d batch=%d seq=%d)", heads, head_dim, batch, seq);
        return (int)cudaErrorInvalidValue;
    }
    if (heads == 0 || batch == 0 || seq == 0) return 0;
    const int sms = current_device_sm_count();
    if (sms <= 0) return (int)cudaErrorNoDevice;
    const __half *hq = static_cast<const __half*>(q), *hk = static_cast<const __half*>(k), *hv = static_cast<const __half*>(v);
    const __half *bq = static_cast<const __half*>(bias_q), *bv = static_cast<const __half*>(bias_v);
    const int64_t tokens = (int64_t)batch * seq;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // Tiles of 128 queries need blocks of keys to pay for their start-up (about 3 us) and are half as many: at 8 heads of 64 tokens 152
    // tiles take 5.8 us against 4.6, at 256 tokens 64 tiles 8.2 (7.8), 128 8.5 (10.2), at 512 tokens 48 tiles 11.9 (13.2).
    const dim3 wide((seq + enc::kTcQueries - 1) / enc::kTcQueries, heads, batch);
    const int64_t tiles = (int64_t)wide.x * heads * batch;
    CUtensorMap tq, tk, tv;
    const bool wanted = kernel == 2 || (kernel == 0 && 2 * tiles * ((seq - 1) / enc::kTile) >= 3 * sms);
    enc::EncodeFn encode = wanted ? enc::encode_fn() : nullptr;
    if (encode && enc::encode_tokens(encode, &tq, q, heads * head_dim, batch, seq) &&
        enc::encode_tokens(encode, &tk, k, heads * head_dim, batch, seq) && enc::encode_tokens(encode, &tv, v, heads * head_dim, batch, seq)) {
        static DeviceOnce once;
        if (!once.done()) {
            const cudaError_t e = cudaFuncSetAttribute(enc::attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, enc::TcSmem::kDynamic);
            if (e != cudaSuccess) { set_error("attention: %s", cudaGetErrorString(e)); return (int)e; }
            once.mark();
        }
        enc::attention_tc_kernel<<<wide, enc::kTcThreads, enc::TcSmem::kDynamic, st>>>(seq, tokens, tq, tk, tv, hq, hk, hv, bq, bv,
                                                                                        static_cast<__half*>(out));
        if (taken) *taken = 2;
    } else if (kernel == 2) {
        set_error("attention: no tensor maps for these operands");
        return (int)cudaErrorNotSupported;
    } else {
        const dim3 grid((seq + enc::kTile - 1) / enc::kTile, heads, batch);
        enc::attention_fm_kernel<<<grid, enc::kAttnThreads, 0, st>>>(seq, tokens, hq, hk, hv, bq, bv, static_cast<__half*>(out));
        if (taken) *taken = 1;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("attention launch: %s", cudaGetErrorString(e)); return (int)e; }
    return 0;
}

}  // extern "C"
