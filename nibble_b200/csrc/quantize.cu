// Group-wise symmetric INT4 quantisation and packing on the device: FP16 or FP32 weights [N, K] ->
// packed codes [N, K/2] + FP16 scales [N, K/group], bit-identical to the reference's host routine
// (w4a16/quantization.py:65-113):
//   step  = amax(|w| over the group) / 7 in FP32, 1 for an all-zero group
//   code  = clamp(round_half_even(w / step), -7, 7)        (FP32 IEEE division, rint)
//   scale = half(step)                                     (rounded after the codes are made)
// Weights that are not finite, whatever the group size: a NaN does not count for the maximum and gets code -7, the other weights
// of its group their own codes; an infinity makes the scale infinite, its own code -7 and those of finite weights 0.
// byte j of a row holds code 2j in its low nibble and code 2j+1 in its high nibble.
//
// Groups of 128, 64 and 32: quantize_pack_group_kernel below, weights read once.
// Other group sizes: one warp per group, weights read twice (maximum, then codes).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "kernels.h"

namespace w4a16 {
namespace {

template <typename T>
__device__ __forceinline__ float load_weight(const T* p);
template <>
__device__ __forceinline__ float load_weight<__half>(const __half* p) { return __half2float(*p); }
template <>
__device__ __forceinline__ float load_weight<float>(const float* p) { return *p; }

__device__ __forceinline__ unsigned code_of(float w, float step) {
    float q = rintf(__fdiv_rn(w, step));
    q = fminf(fmaxf(q, -7.0f), 7.0f);
    return static_cast<unsigned>(static_cast<int>(q)) & 0xFu;
}

template <typename T>
__global__ void __launch_bounds__(256)
quantize_pack_kernel(const T* __restrict__ weights, uint8_t* __restrict__ packed, __half* __restrict__ scales,
                     int64_t total_groups, int group) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); g < total_groups; g += warps) {
        const T* src = weights + g * group;              // groups of a row-major matrix are consecutive in memory
        float amax = 0.0f;
        for (int i = lane; i < group; i += 32) amax = fmaxf(amax, fabsf(load_weight(src + i)));
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, offset));
        const float step = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 7.0f);
        uint8_t* dst = packed + g * (group >> 1);
        if ((group & 3) == 0) {
            for (int q = lane; q < (group >> 2); q += 32) {
                const unsigned c0 = code_of(load_weight(src + 4 * q), step);
                const unsigned c1 = code_of(load_weight(src + 4 * q + 1), step);
                const unsigned c2 = code_of(load_weight(src + 4 * q + 2), step);
                const unsigned c3 = code_of(load_weight(src + 4 * q + 3), step);
                // (g * group / 2 + 2 q) is even: the two bytes are 2-byte aligned when `packed` is
                *reinterpret_cast<uint16_t*>(dst + 2 * q) = static_cast<uint16_t>(c0 | (c1 << 4) | (c2 << 8) | (c3 << 12));
            }
        } else {
            for (int q = lane; q < (group >> 1); q += 32) {
                const unsigned c0 = code_of(load_weight(src + 2 * q), step);
                const unsigned c1 = code_of(load_weight(src + 2 * q + 1), step);
                dst[q] = static_cast<uint8_t>(c0 | (c1 << 4));
            }
        }
        if (lane == 0) scales[g] = __float2half_rn(step);
    }
}

// Eight consecutive weights, as loaded and as floats.
template <typename T>
struct Eight;
template <>
struct Eight<__half> {
    uint4 raw;
    __device__ __forceinline__ void load(const __half* p) { raw = __ldcs(reinterpret_cast<const uint4*>(p)); }
    // largest magnitude: in FP16, two at a time
    __device__ __forceinline__ float amax() const {
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
        const __half2 m = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
        return fmaxf(__low2float(m), __high2float(m));
    }
    __device__ __forceinline__ void floats(float (&w)[8]) const {
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            w[2 * i] = f.x;
            w[2 * i + 1] = f.y;
        }
    }
};
template <>
struct Eight<float> {
    float4 lo, hi;
    __device__ __forceinline__ void load(const float* p) {
        lo = __ldcs(reinterpret_cast<const float4*>(p));
        hi = __ldcs(reinterpret_cast<const float4*>(p) + 1);
    }
    __device__ __forceinline__ float amax() const {
        return fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(lo.z), fabsf(lo.w))),
                     fmaxf(fmaxf(fabsf(hi.x), fabsf(hi.y)), fmaxf(fabsf(hi.z), fabsf(hi.w))));
    }
    __device__ __forceinline__ void floats(float (&w)[8]) const {
        w[0] = lo.x; w[1] = lo.y; w[2] = lo.z; w[3] = lo.w;
        w[4] = hi.x; w[5] = hi.y; w[6] = hi.z; w[7] = hi.w;
    }
};

// The larger of two numbers; NaN if either is.
__device__ __forceinline__ float max_or_nan(float a, float b) {
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}

// Eight codes as one word.
//
// Fast route: t = w * (1/step) + 1.5 * 2^23 in one FMA rounds the exact product to the nearest even integer; r = t - 1.5 * 2^23
// is that integer.  The product and the reference's fl(w / step) differ by a few ulp at most, so both round to the same
// integer unless the quotient sits within 1e-4 of a tie k + 0.5; a lane that sees such a weight (about one in 600) redoes its
// codes with the IEEE division.
//
// Packing in floats: four codes are a number of at most 16 bits, r0 + 16 r1 + 256 r2 + 4096 r3 + 0x8888, exact in FP32 and read
// off the mantissa after adding 2^23; the 8 added to each nibble is its sign bit flipped.  A weight that is infinite or NaN, or
// a 1/step that is infinite, would spoil all four codes; it makes its distance from r NaN, which the maximum passes on (fmaxf
// would drop it), and the division gives each weight its own code.  (Looking at the packed sums
// instead, 28672 x 8192 from FP16: 122 -> 126 us; this way no change.)
__device__ __forceinline__ uint32_t pack_codes(const float (&w)[8], float step, float inv_step) {
    constexpr float kMagic = 12582912.0f;
    float r[8], off = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        r[i] = fmaf(w[i], inv_step, kMagic) - kMagic;
        off = max_or_nan(off, fabsf(fmaf(w[i], inv_step, -r[i])));
    }
    const float lo = fmaf(fmaf(fmaf(r[3], 16.0f, r[2]), 16.0f, r[1]), 16.0f, r[0]) + (8388608.0f + 34952.0f);
    const float hi = fmaf(fmaf(fmaf(r[7], 16.0f, r[6]), 16.0f, r[5]), 16.0f, r[4]) + (8388608.0f + 34952.0f);
    uint32_t word = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x5410) ^ 0x88888888u;
    if (!(off <= 0.4999f)) {
        word = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) word |= code_of(w[i], step) << (4 * i);
    }
    return word;
}

// GROUP 128, 64 or 32 and 16-byte aligned weights: GROUP / 16 lanes share a group, a lane holds weights 8l..8l+7 of each half
// of it, so both loads of the lanes are contiguous, and what a group costs once (two IEEE divisions, the shuffles) is
// shared by 16 weights.  Bound: HBM at 2.5 bytes (FP16) or 4.5 (FP32) a weight, with about nine instructions a weight close behind.
// 28672 x 8192 from FP16, 128-wide groups: 148 -> 109 us (5.4 TB/s);
// from FP32 155 us (6.8 TB/s); with 64- and 32-wide groups, which read the weights twice before, 803 and 1406 -> 115 us.
// Eight blocks per SM for FP16 (32 registers) and as many blocks as there are groups for FP32: 114 -> 109 us and 164 -> 155.
template <typename T, int GROUP>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 8 : 6)
quantize_pack_group_kernel(const T* __restrict__ weights, uint8_t* __restrict__ packed, __half* __restrict__ scales,
                           int64_t total_groups) {
    constexpr int kLanes = GROUP / 16;
    constexpr int kGroupsPerBlock = 256 / kLanes;
    const int l = threadIdx.x % kLanes;
    for (int64_t block = blockIdx.x; block * kGroupsPerBlock < total_groups; block += gridDim.x) {
        const int64_t g = block * kGroupsPerBlock + threadIdx.x / kLanes;
        const bool live = g < total_groups;
        Eight<T> a, b;
        const T* src = weights + (live ? g : total_groups - 1) * GROUP + l * 8;
        a.load(src);
        b.load(src + GROUP / 2);
        float amax = fmaxf(fmaxf(a.amax(), b.amax()), 0.0f);     // 0 where every weight is NaN
#pragma unroll
        for (int offset = kLanes / 2; offset > 0; offset >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, offset));
        const float step = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 7.0f);
        const float inv_step = __fdiv_rn(1.0f, step);
        float w[8];
        uint32_t* out = reinterpret_cast<uint32_t*>(packed + g * (GROUP / 2)) + l;
        a.floats(w);
        const uint32_t first = pack_codes(w, step, inv_step);
        b.floats(w);
        const uint32_t second = pack_codes(w, step, inv_step);
        if (live) {
            out[0] = first;
            out[GROUP / 16] = second;
            if (l == 0) scales[g] = __float2half_rn(step);
        }
    }
}

template <typename T>
int launch(const T* weights, uint8_t* packed, __half* scales, int64_t N, int64_t K, int64_t group, cudaStream_t stream) {
    const int64_t total_groups = N * (K / group);
    if ((group == 128 || group == 64 || group == 32) && reinterpret_cast<uintptr_t>(weights) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(packed) % 4 == 0) {
        const int64_t groups_per_block = 256 / (group / 16);
        const int64_t fast_blocks = std::min<int64_t>((total_groups + groups_per_block - 1) / groups_per_block,
                                                           sizeof(T) == 2 ? 148 * 64 : INT32_MAX);
        const auto kernel = group == 128 ? quantize_pack_group_kernel<T, 128>
                            : group == 64 ? quantize_pack_group_kernel<T, 64> : quantize_pack_group_kernel<T, 32>;
        kernel<<<static_cast<unsigned>(fast_blocks), 256, 0, stream>>>(weights, packed, scales, total_groups);
        if (cudaGetLastError() != cudaSuccess) return W4A16_ERR_LAUNCH;
        g_launch_count.fetch_add(1, std::memory_order_relaxed);
        return W4A16_OK;
    }
    const int64_t blocks = std::min<int64_t>((total_groups + 7) / 8, 148 * 64);
    quantize_pack_kernel<T><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(weights, packed, scales, total_groups,
                                                                              static_cast<int>(group));
    if (cudaGetLastError() != cudaSuccess) return W4A16_ERR_LAUNCH;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return W4A16_OK;
}

}  // namespace

int launch_quantize_pack(const void* weights, bool is_f32, uint8_t* packed, __half* scales, int64_t N, int64_t K,
                         int64_t group, cudaStream_t stream) {
    if (is_f32) return launch(static_cast<const float*>(weights), packed, scales, N, K, group, stream);
    return launch(static_cast<const __half*>(weights), packed, scales, N, K, group, stream);
}

}  // namespace w4a16
