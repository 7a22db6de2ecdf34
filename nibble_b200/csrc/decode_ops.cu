// The small kernels either side of the linear layers in one LLaMA decode step (batch 1), so that a
// token is ~8 launches per decoder block instead of the several dozen elementwise kernels a
// framework issues:
//   add_rmsnorm   residual add (FP16) + RMSNorm with FP32 statistics          -> input of q/k/v or gate/up
//   attention     RoPE on q and k, append k/v to the cache, softmax(q k^T / sqrt(d)) v over the cache
//   silu_mul      silu(gate) * up on the fused gate/up output                   -> input of down_proj
// They restate what the reference's generation script gets from HuggingFace's LlamaDecoderLayer
// (scripts/generate.py:260-365 drives model.generate; the arithmetic is transformers' modeling_llama:
// LlamaRMSNorm, apply_rotary_pos_emb / rotate_half, scaled dot product attention with grouped KV heads,
// LlamaMLP).  Roundings follow that code: the residual sum, the normalised value, the rotary
// products and silu(gate) are each rounded to FP16 where the framework rounds them.
//
// The position is read from device memory, so one captured graph serves every step.
//
// Every kernel releases its successor at once (griddepcontrol.launch_dependents) and waits for its
// predecessor (griddepcontrol.wait) before it touches memory: when launched with the programmatic
// attribute, the next kernel's blocks are resident and -- for the linears -- already streaming weights
// while this one computes.  Both instructions do nothing under an ordinary launch.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "unpack.cuh"

namespace w4a16 {
namespace {

__device__ __forceinline__ float block_sum(float v, float* scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    __syncthreads();                       // scratch may still be read from a previous call
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = 0.0f;
    for (int w = 0; w < warps; ++w) total += scratch[w];
    return total;
}

// stream_out = half(stream_in + delta) (or stream_in when delta is null); normed = weight * half(s * rsqrt(mean(s^2) + eps))
__global__ void __launch_bounds__(256)
add_rmsnorm_kernel(const __half* __restrict__ stream_in, const __half* __restrict__ delta, const __half* __restrict__ weight,
                   __half* __restrict__ stream_out, __half* __restrict__ normed, int hidden, float eps) {
    __shared__ float scratch[8];
    extern __shared__ __half row[];        // the summed stream, kept for the second pass
    pdl_release_downstream();
    pdl_wait_for_upstream();
    float sq = 0.0f;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        __half s = stream_in[i];
        if (delta != nullptr) s = __hadd(s, delta[i]);
        row[i] = s;
        const float f = __half2float(s);
        sq += f * f;
    }
    const float inv = rsqrtf(block_sum(sq, scratch) / static_cast<float>(hidden) + eps);
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        const __half s = row[i];
        if (stream_out != nullptr) stream_out[i] = s;
        normed[i] = __hmul(weight[i], __float2half_rn(__half2float(s) * inv));
    }
}

__global__ void __launch_bounds__(256)
silu_mul_kernel(const __half* __restrict__ gate_up, __half* __restrict__ out, int inter) {
    pdl_release_downstream();
    pdl_wait_for_upstream();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= inter) return;
    const __half2 act = silu_half2(__half2half2(gate_up[i]));
    out[i] = __hmul(__low2half(act), gate_up[inter + i]);
}

// token = index of the first largest logit (what argmax returns); the position moves on by one.
__global__ void __launch_bounds__(1024)
argmax_advance_kernel(const __half* __restrict__ logits, int count, long long* __restrict__ token,
                      long long* __restrict__ position) {
    __shared__ float best_value[32];
    __shared__ int best_index[32];
    pdl_release_downstream();
    pdl_wait_for_upstream();
    float value = -INFINITY;
    int index = 0x7fffffff;
    for (int i = threadIdx.x * 8; i < count; i += blockDim.x * 8) {
        if (i + 8 <= count && (reinterpret_cast<uintptr_t>(logits + i) & 15) == 0) {
            const uint4 q = *reinterpret_cast<const uint4*>(logits + i);
            const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __half22float2(h[j]);
                if (f.x > value) { value = f.x; index = i + 2 * j; }
                if (f.y > value) { value = f.y; index = i + 2 * j + 1; }
            }
        } else {
            for (int j = i; j < min(i + 8, count); ++j) {
                const float f = __half2float(logits[j]);
                if (f > value) { value = f; index = j; }
            }
        }
    }
    auto merge = [&](float other_value, int other_index) {
        if (other_value > value || (other_value == value && other_index < index)) { value = other_value; index = other_index; }
    };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) merge(__shfl_xor_sync(0xffffffffu, value, o), __shfl_xor_sync(0xffffffffu, index, o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { best_value[warp] = value; best_index[warp] = index; }
    __syncthreads();
    if (warp == 0) {
        const int warps = blockDim.x >> 5;
        value = lane < warps ? best_value[lane] : -INFINITY;
        index = lane < warps ? best_index[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) merge(__shfl_xor_sync(0xffffffffu, value, o), __shfl_xor_sync(0xffffffffu, index, o));
        if (lane == 0) {
            *token = index == 0x7fffffff ? 0 : index;
            if (position != nullptr) *position += 1;
        }
    }
}

struct AttentionParams {
    const __half* qkv;        // [q heads * d | kv heads * d | kv heads * d] of this token
    __half* k_cache;          // [kv heads][max_len][d]
    __half* v_cache;
    __half* out;              // [q heads * d]
    const long long* position;  // device scalar: index of this token
    const float* inv_freq;    // [d / 2]
    int q_heads, kv_heads, head_dim, max_len;
    float rope_scale;         // multiplies cos and sin (1 for plain RoPE)
    float softmax_scale;
    unsigned* status;         // set to 1 when the position does not fit the cache
};

// A cluster of CTAs per query head; each CTA takes a contiguous part of the cached positions, and every group of D/8 lanes
// walks its own positions with a running maximum, sum and weighted V row, so nothing is exchanged before the end.  Then
// the warps of a CTA are added up in shared memory, each CTA's result is written into the first CTA's shared memory
// (distributed shared memory), one cluster barrier, and the first CTA adds those up.
//
// Bound: latency of a dependent kernel at short contexts, loads in flight at long ones.  One CTA per head left 116 SMs idle
// and took 47.6 us a layer at 1500 positions (TinyLlama: 32 heads of 64); four take 5.4 us.  Two or four heads of a KV
// head in one CTA would read each K and V row fewer times out of L2; it was 0.4 us faster there and 0.5 us slower at 4
// positions, where the extra arithmetic is all latency.  Eight passes are requested ahead (two register buffers of
// kAttnBatch rows of K and V), and the grid stays at one CTA per SM: with four passes and twice the CTAs a TinyLlama token
// took 530 us at 1500 positions, 504 at 500 and 454 at 4, against 518, 470 and 444.  Contexts of one part's worth use one CTA per cluster and no cluster barrier: the other
// CTAs leave at once.
constexpr int kAttnThreads = 256;
constexpr int kAttnWarps = kAttnThreads / 32;
constexpr int kAttnMaxParts = 8;                      // CTAs per cluster: the portable limit
constexpr int kAttnBatch = 4;                         // passes requested together
constexpr float kNoScore = -1.0e30f;

__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_acquire() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// The address of `local` in the shared memory of the cluster's first CTA.
__device__ __forceinline__ uint32_t in_first_cta(const void* local) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(local))));
    return remote;
}
__device__ __forceinline__ void store_cluster(uint32_t address, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(address), "f"(v) : "memory");
}

// Eight FP16 values of the token's qkv row, which need not start on a 16-byte boundary.
__device__ __forceinline__ uint4 load8_any(const __half* src) {
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) return *reinterpret_cast<const uint4*>(src);
    uint4 q;
    __half* h = reinterpret_cast<__half*>(&q);
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = src[i];
    return q;
}

// Rotary embedding of eight dims, rounded as the framework rounds it: cos/sin in FP16, two FP16 products, one FP16 sum
// (the _rn forms are never contracted into one fused multiply-add).  `own` holds the dims, `other` the ones half a head away.
__device__ __forceinline__ uint4 rotate8(const uint4& own, const uint4& other, bool first_half, const __half2* c, const __half2* s) {
    uint4 out;
    const __half2* a = reinterpret_cast<const __half2*>(&own);
    const __half2* b = reinterpret_cast<const __half2*>(&other);
    __half2* o = reinterpret_cast<__half2*>(&out);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 turned = first_half ? __hneg2(b[i]) : b[i];
        o[i] = __hadd2_rn(__hmul2_rn(a[i], c[i]), __hmul2_rn(turned, s[i]));
    }
    return out;
}

template <int D>
__global__ void __launch_bounds__(kAttnThreads)
attention_decode_kernel(const AttentionParams p) {
    constexpr int kLanesPerPos = D / 8;
    constexpr int kPosPerPass = kAttnThreads / kLanesPerPos;   // 32 (D = 64) or 16 (D = 128)
    constexpr int kPosPerBatch = kPosPerPass * kAttnBatch;
    constexpr int kPosPerPart = 4 * kPosPerPass;               // at least: less is not worth the cluster barrier
    constexpr int half_d = D / 2;
    __shared__ __align__(16) __half cos_table[half_d];
    __shared__ __align__(16) __half sin_table[half_d];
    static_assert(D <= kAttnThreads);
    __shared__ __align__(16) float warp_acc[kAttnWarps][D];
    __shared__ float warp_max[kAttnWarps], warp_sum[kAttnWarps];
    __shared__ float part_acc[kAttnMaxParts][D];               // the first CTA's are written by the whole cluster
    __shared__ float part_max[kAttnMaxParts], part_sum[kAttnMaxParts];

    uint32_t part, max_parts;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(part));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(max_parts));
    const int head = blockIdx.x / max_parts;
    const int group_heads = p.q_heads / p.kv_heads;
    const int kv_head = head / group_heads;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = tid % kLanesPerPos;               // which 8 of the D dims
    const int slot = tid / kLanesPerPos;              // which position of a pass
    pdl_release_downstream();
    // Nothing up to the wait depends on the kernel just before this one (it produces qkv): the position was set and the
    // older cache rows were written by earlier steps.  The first part starts at position 0 whatever the context, so its
    // first rows are requested without waiting for the position; rows past it hold stale data and are never used.
    const long long pos = *p.position;
    const float freq = p.inv_freq[tid % half_d];
    const size_t head_base = static_cast<size_t>(kv_head) * p.max_len * kLanesPerPos + sub;
    const uint4* k_rows = reinterpret_cast<const uint4*>(p.k_cache) + head_base;
    const uint4* v_rows = reinterpret_cast<const uint4*>(p.v_cache) + head_base;
    struct Rows {
        uint4 k[kAttnBatch], v[kAttnBatch];
    };
    Rows even, odd;
    if (part == 0) {
        const size_t t = static_cast<size_t>(min(slot, p.max_len - 1));
        even.k[0] = k_rows[t * kLanesPerPos];
        even.v[0] = v_rows[t * kLanesPerPos];
    }
    if (pos < 0 || pos >= p.max_len) {
        if (tid == 0 && part == 0) atomicMax(p.status, 1u);
        pdl_wait_for_upstream();
        return;
    }
    const int newest = static_cast<int>(pos);         // positions [0, newest) come from the cache, the newest from qkv
    const int parts = min(static_cast<int>(max_parts), newest / kPosPerPart + 1);
    if (parts == 1 && part > 0) return;
    if (parts > 1) cluster_arrive_relaxed();          // "this CTA runs": waited for before its memory is written to
    if (static_cast<int>(part) >= parts) {            // no positions for this CTA: it only takes part in the barriers
        cluster_wait_acquire();
        cluster_arrive_release();
        cluster_wait_acquire();
        return;
    }
    const int per_part = newest / parts + 1;
    const int begin = static_cast<int>(part) * per_part;
    const int end = min(newest + 1, begin + per_part);
    auto fetch = [&](Rows& rows, int base) {
#pragma unroll
        for (int e = 0; e < kAttnBatch; ++e) {
            const int t = base + e * kPosPerPass + slot;
            if (t < min(end, newest) && (e > 0 || base > 0)) {
                rows.k[e] = k_rows[static_cast<size_t>(t) * kLanesPerPos];
                rows.v[e] = v_rows[static_cast<size_t>(t) * kLanesPerPos];
            }
        }
    };
    fetch(even, begin);
    fetch(odd, begin + kPosPerBatch);
    if (tid < half_d) {
        float sn, cs;
        sincosf(static_cast<float>(pos) * freq, &sn, &cs);
        cos_table[tid] = __float2half_rn(cs * p.rope_scale);
        sin_table[tid] = __float2half_rn(sn * p.rope_scale);
    }
    __syncthreads();
    const bool first_half = sub < kLanesPerPos / 2;
    const int pair_sub = sub ^ (kLanesPerPos / 2);    // the lane whose dims are half a head away
    const __half2* my_cos = reinterpret_cast<const __half2*>(cos_table + (sub * 8) % half_d);
    const __half2* my_sin = reinterpret_cast<const __half2*>(sin_table + (sub * 8) % half_d);

    pdl_wait_for_upstream();
    const __half* q_in = p.qkv + head * D;
    const __half* k_in = p.qkv + p.q_heads * D + kv_head * D;
    const __half* v_in = p.qkv + (p.q_heads + p.kv_heads) * D + kv_head * D;
    const uint4 q_own = load8_any(q_in + sub * 8), q_other = load8_any(q_in + pair_sub * 8);
    uint4 k_new = make_uint4(0u, 0u, 0u, 0u), v_new = k_new;
    if (end > newest) {                               // the CTA whose part ends with the newest position
        const uint4 k_own = load8_any(k_in + sub * 8), k_other = load8_any(k_in + pair_sub * 8);
        v_new = load8_any(v_in + sub * 8);
        k_new = rotate8(k_own, k_other, first_half, my_cos, my_sin);
        if (slot == 0 && head % group_heads == 0) {   // one cluster of the KV head appends to the cache
            const size_t row = head_base + static_cast<size_t>(newest) * kLanesPerPos;
            reinterpret_cast<uint4*>(p.k_cache)[row] = k_new;
            reinterpret_cast<uint4*>(p.v_cache)[row] = v_new;
        }
    }
    auto widen8 = [](const uint4& piece, float (&f)[8]) {
        const __half2* pairs = reinterpret_cast<const __half2*>(&piece);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 two = __half22float2(pairs[i]);
            f[2 * i] = two.x;
            f[2 * i + 1] = two.y;
        }
    };
    float q[8], acc[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float top = kNoScore, sum = 0.0f;
    widen8(rotate8(q_own, q_other, first_half, my_cos, my_sin), q);
    auto use = [&](Rows& rows, int base) {
        if (base + warp * (32 / kLanesPerPos) >= end) return;   // nothing for this warp
        float dot[kAttnBatch];
#pragma unroll
        for (int e = 0; e < kAttnBatch; ++e) {
            float k[8];
            widen8(base + e * kPosPerPass + slot == newest ? k_new : rows.k[e], k);
            dot[e] = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) dot[e] += q[i] * k[i];
        }
#pragma unroll
        for (int o = kLanesPerPos / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int e = 0; e < kAttnBatch; ++e) dot[e] += __shfl_xor_sync(0xffffffffu, dot[e], o);
        }
        // a new maximum: what has been summed so far shrinks by e^(old - new)
        float next = top;
#pragma unroll
        for (int e = 0; e < kAttnBatch; ++e) {
            dot[e] *= p.softmax_scale;
            if (base + e * kPosPerPass + slot < end) next = fmaxf(next, dot[e]);
        }
        const float shrink = expf(top - next);
        top = next;
        sum *= shrink;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] *= shrink;
#pragma unroll
        for (int e = 0; e < kAttnBatch; ++e) {
            const int t = base + e * kPosPerPass + slot;
            if (t < end) {
                float v[8];
                widen8(t == newest ? v_new : rows.v[e], v);
                const float w = expf(dot[e] - top);
                sum += w;
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] += w * v[i];
            }
        }
    };
    for (int base = begin; base < end; base += 2 * kPosPerBatch) {
        use(even, base);
        fetch(even, base + 2 * kPosPerBatch);
        use(odd, base + kPosPerBatch);
        fetch(odd, base + 3 * kPosPerBatch);
    }
    // lane groups of a warp, then the warps, then the CTAs of the cluster
#pragma unroll
    for (int o = kLanesPerPos; o < 32; o <<= 1) {
        const float other_top = __shfl_xor_sync(0xffffffffu, top, o);
        const float next = fmaxf(top, other_top);
        const float mine = expf(top - next), theirs = expf(other_top - next);
        top = next;
        sum = sum * mine + __shfl_xor_sync(0xffffffffu, sum, o) * theirs;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = acc[i] * mine + __shfl_xor_sync(0xffffffffu, acc[i], o) * theirs;
    }
    if (lane < kLanesPerPos) {
        float4* to = reinterpret_cast<float4*>(&warp_acc[warp][lane * 8]);
        to[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        to[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        if (lane == 0) {
            warp_max[warp] = top;
            warp_sum[warp] = sum;
        }
    }
    __syncthreads();
    // one element of the head's output: its weighted sum, the sum of the weights, and the maximum both refer to
    auto merge = [&](int count, const float* maxima, const float* sums, const float (*rows)[D], float& best, float& total,
                     float& weight) {
        best = kNoScore;
        total = weight = 0.0f;
        for (int r = 0; r < count; ++r) best = fmaxf(best, maxima[r]);
        for (int r = 0; r < count; ++r) {
            const float w = expf(maxima[r] - best);
            weight += w * sums[r];
            total += w * rows[r][tid];
        }
    };
    float best, total, weight;
    if (parts > 1) cluster_wait_acquire();            // every CTA of the cluster has started
    if (tid < D) {
        merge(kAttnWarps, warp_max, warp_sum, warp_acc, best, total, weight);
        if (parts == 1) {
            p.out[head * D + tid] = __float2half_rn(total / weight);
        } else {
            store_cluster(in_first_cta(&part_acc[part][tid]), total);
            if (tid == 0) {
                store_cluster(in_first_cta(&part_max[part]), best);
                store_cluster(in_first_cta(&part_sum[part]), weight);
            }
        }
    }
    if (parts == 1) return;
    __syncwarp();
    cluster_arrive_release();
    cluster_wait_acquire();
    if (part == 0 && tid < D) {
        merge(parts, part_max, part_sum, part_acc, best, total, weight);
        p.out[head * D + tid] = __float2half_rn(total / weight);
    }
}

template <typename... Params, typename... Args>
int launch_kernel(void (*kernel)(Params...), dim3 grid, dim3 block, int cluster, size_t smem, bool programmatic,
                  cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t launch = {};
    launch.gridDim = grid;
    launch.blockDim = block;
    launch.dynamicSmemBytes = smem;
    launch.stream = stream;
    cudaLaunchAttribute attr[2];
    launch.attrs = attr;
    if (programmatic) {
        attr[launch.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[launch.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[launch.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[launch.numAttrs].val.clusterDim.x = static_cast<unsigned>(cluster);
        attr[launch.numAttrs].val.clusterDim.y = 1;
        attr[launch.numAttrs++].val.clusterDim.z = 1;
    }
    if (cudaLaunchKernelEx(&launch, kernel, static_cast<Params>(args)...) != cudaSuccess) return W4A16_ERR_LAUNCH;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return W4A16_OK;
}

}  // namespace

int launch_add_rmsnorm(const __half* stream_in, const __half* delta, const __half* weight, __half* stream_out,
                       __half* normed, int hidden, float eps, bool programmatic, cudaStream_t stream) {
    return launch_kernel(add_rmsnorm_kernel, dim3(1), dim3(256), 1, static_cast<size_t>(hidden) * sizeof(__half), programmatic,
                         stream, stream_in, delta, weight, stream_out, normed, hidden, eps);
}

int launch_silu_mul(const __half* gate_up, __half* out, int inter, bool programmatic, cudaStream_t stream) {
    return launch_kernel(silu_mul_kernel, dim3((inter + 255) / 256), dim3(256), 1, 0, programmatic, stream, gate_up, out, inter);
}

int launch_argmax_advance(const __half* logits, int count, long long* token, long long* position, bool programmatic,
                          cudaStream_t stream) {
    return launch_kernel(argmax_advance_kernel, dim3(1), dim3(1024), 1, 0, programmatic, stream, logits, count, token, position);
}

int launch_attention_decode(const __half* qkv, __half* k_cache, __half* v_cache, __half* out, const long long* position,
                            const float* inv_freq, int q_heads, int kv_heads, int head_dim, int max_len, float rope_scale,
                            float softmax_scale, unsigned* status, bool programmatic, cudaStream_t stream) {
    AttentionParams params{qkv, k_cache, v_cache, out, position, inv_freq, q_heads, kv_heads, head_dim, max_len,
                           rope_scale, softmax_scale, status};
    auto kernel = head_dim == 64 ? attention_decode_kernel<64> : attention_decode_kernel<128>;
    // CTAs per head: as many as the cache can give a part's worth of positions each, and no more than one per SM in all.
    const int positions = kAttnThreads / (head_dim / 8) * 4;
    int parts = 1;
    while (parts < kAttnMaxParts && parts * positions < max_len && 2 * parts * q_heads <= 148) parts *= 2;
    return launch_kernel(kernel, dim3(static_cast<unsigned>(q_heads) * parts), dim3(kAttnThreads), parts, 0, programmatic,
                         stream, params);
}

}  // namespace w4a16
