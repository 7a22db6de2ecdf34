// extern "C" boundary of libw4a16_b200: argument validation and kernel routing only.
// The declarations, their contracts and the reference functions they replace are in
// include/w4a16_b200.h.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"

namespace w4a16 {
std::atomic<uint64_t> g_launch_count{0};
}

namespace {

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

int validate_linear(const void* x, const void* packed, const void* scales, const void* y, int64_t M,
                    int64_t N, int64_t K, int64_t group) {
    if (M < 0 || N < 0 || K < 0 || (K & 1)) return W4A16_ERR_BAD_SHAPE;
    if (group <= 0 || (group & 1)) return W4A16_ERR_BAD_GROUP;
    if (K % group != 0) return W4A16_ERR_BAD_SHAPE;
    if (M == 0 || N == 0) return W4A16_OK;
    if (y == nullptr) return W4A16_ERR_NULL_POINTER;
    if (K > 0 && (x == nullptr || packed == nullptr || scales == nullptr)) return W4A16_ERR_NULL_POINTER;
    return W4A16_OK;
}

bool fast_path_applies(const void* x, const void* packed, int64_t K, int64_t group) {
    return group == w4a16::kGroupFast && K > 0 && aligned16(x) && aligned16(packed);
}

// Groups below 128 stream like 128-wide ones while K still comes in whole 128-wide chunks.
bool small_group_streams(const void* x, const void* packed, const void* scales, int64_t K, int64_t group) {
    return group != w4a16::kGroupFast && w4a16::is_stream_group(group) && K > 0 && K % w4a16::kGroupFast == 0 && aligned16(x) &&
           aligned16(packed) && aligned16(scales);
}

}  // namespace

namespace {

// Ranges of K that CTAs would share a 128 x 256 tile in: up to four where half the SMs or more would idle, of 1024 and more.  Part
// of the line below; and of the workspace query, whose answer also serves explicit launch shapes that split K.  The GEMMs share tiles
// in ways of their own, which w4a16_linear_scratch_bytes knows.
int k_ranges(int64_t M, int64_t N, int64_t K) {
    const int64_t tiles = (M + 255) / 256 * ((N + 127) / 128);
    int64_t ranges = tiles > 0 ? std::min<int64_t>(4, 148 / tiles) : 1;
    ranges = std::max<int64_t>(1, std::min<int64_t>(ranges, K / (K >= 4096 ? 1024 : 2048)));
    const int64_t width = ((K + ranges - 1) / ranges + 255) / 256 * 256;
    return static_cast<int>((K + width - 1) / width);
}

// Whether a fast-path call with FP16 output goes to a GEMM rather than the streaming kernel: from 65 rows on always, up to 8 rows
// never.  Between 9 and 64 the line decides the arithmetic as well as the time: the streaming kernel multiplies exact codes and
// scales its FP32 sums, the GEMM rounds each weight to FP16 first.  So the line stays where it was drawn, and no batch that has
// exact weights loses them to a faster kernel.  It was drawn from the cost of the GEMM with weights in shared memory (0.6 us per
// 128-wide K step of a round of 148 tiles, 3 us for sharing K) against the streaming kernel's (5 us plus 8 + 1.5 * K/1024 us
// per 1e9 multiply-adds of the batch padded to 32 or 64 rows) -- these are the constants below; the calls it sends on run the
// faster GEMM of linear_gemm.cu.
// Measured on 23 layers at nine batches (us, streaming / that GEMM): beyond the line the GEMM is never slower by more than 5 % (14336 ->
// 4096, 9 rows: 17.9 / 18.9) and up to six times as fast (8192 -> 28672, 64 rows: 251 / 47); on this side of it exact weights are
// faster on small layers (2048 x 2048, 32 rows: 7.2 / 7.9) and cost up to twice the time on others (8192 -> 28672, 16 rows:
// 70 / 41; 3072 -> 8192, 32 rows: 24.9 / 11.7).
bool routes_to_tcgen05(int64_t M, int64_t N, int64_t K, uint32_t flags) {
    if (flags & (W4A16_FLAG_OUTPUT_F32 | W4A16_FLAG_NO_TCGEN05 | W4A16_FLAG_FORCE_GENERIC)) return false;
    if ((flags & W4A16_FLAG_FORCE_TCGEN05) || M >= w4a16::kTcgen05MinRows) return true;
    if (M <= 8) return false;
    // Narrow layers, which those costs do not describe: from 17 rows on, when a fourth of K is what fits the streaming kernel's
    // shared memory and the layer has eight weight tiles (from 33 rows on below N = 2048).  5632 -> 2048, 32 rows: 16.0 / 10.8.
    if (N < 4096) return M > 16 && N >= 1024 && K >= 4992 && (N >= 2048 || M > 32);
    const double padded = M <= 16 ? 16.0 : M <= 32 ? 32.0 : 64.0;
    const double giga_macs = padded * static_cast<double>(K) * static_cast<double>(N) * 1e-9;
    const double streaming_us = 5.0 + giga_macs * (8.0 + 1.5 * static_cast<double>(K) / 1024.0);
    const int64_t rounds = ((N + 127) / 128 + 147) / 148;
    const int ranges = k_ranges(M, N, K);
    const double gemm_us = 3.5 + 0.6 * static_cast<double>(rounds) * static_cast<double>(K) / (128.0 * ranges) + (ranges > 1 ? 3.0 : 0.0);
    // 9..16 rows are close to the streaming kernel's best case: only a clear win moves them
    return gemm_us < (M <= 16 ? 0.85 : 1.0) * streaming_us;
}

// Whether a call that goes to a GEMM takes the one on pairs of SMs, with whole tiles of 256 weight rows x up to 256 batch rows, or the
// one on single SMs, with up to 128 batch rows a tile and the K of few tiles shared, which for some layers takes a workspace.  By their
// models' times for what either would do (us, pairs / single SMs:
// 8192 -> 28672, 2048 rows 730 to 740 / 910 to 1060; 8192 x 8192, 512 rows 59 / 67; 5632 -> 2048, 777 rows 30 / 24), with two lines:
//   - up to 128 rows, one batch tile of the second kernel, only in one round of pairs: in two it loses (8192 -> 28672, 96 rows:
//     63 / 55; in one, 1024 -> 8192, 128 rows: 7.0 / 10.4);
//   - above 512 rows the second kernel only where its tiles fit a round, two with K >= 4096, or K >= 2048 up to 1024 rows: beyond,
//     the first is the faster one whatever the models say (157 calls, at most 1 % slower).
bool gemm_on_pairs(int64_t M, int64_t N, int64_t K, size_t workspace_bytes) {
    if (M <= 64 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) return false;     // (9 to 64 rows, and whatever a flag sends)
    if (M <= 128 && w4a16::gemm_pair_rounds(M, N) != 1) return false;
    const int64_t tiles = (N + 255) / 256 * ((M + 127) / 128);
    if (M > 512 && tiles > 148 && !(tiles <= 296 && K >= 4096) && !(M <= 1024 && K >= 2048)) return true;
    return w4a16::gemm_pair_time(M, N, K) < w4a16::gemm_time(M, N, K, workspace_bytes);
}

int launch_gemm(const w4a16::LinearProblem& p, cudaStream_t stream) {
    const bool pairs = gemm_on_pairs(p.M, p.N, p.K, w4a16::usable_workspace(p));
    return pairs ? w4a16::launch_linear_gemm_pair(p, stream) : w4a16::launch_linear_gemm(p, stream);
}

// Whether a call with 64- or 32-wide groups goes to the GEMM, which rounds each weight to FP16.  Only where the caller has said
// that this will do (as the module does, which dequantises to FP16 above 64 rows in any case): the operator's contract for these
// groups is exact codes and FP32 scales whatever the batch.
bool small_group_routes_to_gemm(int64_t M, uint32_t flags) {
    if (flags & W4A16_FLAG_OUTPUT_F32) return false;
    if (flags & W4A16_FLAG_FORCE_TCGEN05) return true;
    return (flags & W4A16_FLAG_FP16_WEIGHTS) && !(flags & W4A16_FLAG_NO_TCGEN05) && M >= w4a16::kTcgen05MinRows;
}

// Batch rows of one launch where a larger batch of small groups streams: two passes of the kernel, side by side.
constexpr int64_t kSmallGroupRows = 64;

// The streaming kernel, with K split across CTAs only as far as the caller's workspace allows.
int launch_streaming(const w4a16::LinearProblem& p, bool small_group, uint32_t flags, cudaStream_t stream) {
    const bool out_f32 = (flags & W4A16_FLAG_OUTPUT_F32) != 0;
    int max_splits = 1;
    if (p.workspace != nullptr && aligned16(p.workspace)) {
        for (int splits = w4a16::kMaxKSplits; splits > 1; splits >>= 1) {
            if (p.workspace_bytes >= w4a16::linear_workspace_bytes_for(p.M, p.N, splits)) {
                max_splits = splits;
                break;
            }
        }
    }
    w4a16_linear_config cfg = w4a16::choose_linear_config(p.M, p.N, p.K, max_splits, small_group);
    if (reinterpret_cast<uintptr_t>(p.scales) % 4 != 0) cfg.unroll = 1;
    const int launched = w4a16::launch_linear_mma(p, cfg, (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0, out_f32, stream);
    // Too much activation data for one CTA's shared memory and no workspace to split K further: the tcgen05 GEMM
    // has no such limit (nor has the generic kernel, for FP32 output, small groups or when the GEMM is switched off).
    if (launched != W4A16_ERR_WORKSPACE) return launched;
    if (!out_f32 && !small_group && !(flags & W4A16_FLAG_NO_TCGEN05)) return launch_gemm(p, stream);
    return w4a16::launch_linear_generic(p, out_f32, stream);
}

}  // namespace

bool w4a16::linear_routes_to_tcgen05(int64_t M, int64_t N, int64_t K, uint32_t flags) {
    return routes_to_tcgen05(M, N, K, flags);
}

extern "C" {

int w4a16_abi_version(void) { return 2; }

uint64_t w4a16_launch_count(void) { return w4a16::g_launch_count.load(std::memory_order_relaxed); }

const char* w4a16_status_string(int status) {
    switch (status) {
        case W4A16_OK: return "ok";
        case W4A16_ERR_NULL_POINTER: return "a required pointer is NULL";
        case W4A16_ERR_BAD_SHAPE: return "invalid shape: sizes must be non-negative, K even and divisible by group_size";
        case W4A16_ERR_BAD_GROUP: return "invalid group_size for this entry point";
        case W4A16_ERR_MISALIGNED: return "a pointer misses the required 16-byte alignment";
        case W4A16_ERR_WORKSPACE: return "workspace missing or too small";
        case W4A16_ERR_BAD_CONFIG: return "launch configuration not available";
        case W4A16_ERR_LAUNCH: return "CUDA kernel launch failed";
        case W4A16_ERR_TOO_LARGE: return "problem size exceeds what this entry point supports";
        default: return "unknown status";
    }
}

size_t w4a16_linear_workspace_bytes_flags(int64_t M, int64_t N, int64_t K, uint32_t flags) {
    if (M <= 0 || N <= 0 || K <= 0 || K % w4a16::kGroupFast != 0 || (flags & W4A16_FLAG_FORCE_GENERIC)) return 0;
    size_t wanted;
    if (routes_to_tcgen05(M, N, K, flags)) {
        wanted = w4a16::linear_workspace_bytes_for(M, N, k_ranges(M, N, K));
    } else {
        // a layer of few row tiles and long K may always be split, if only by w4a16_linear_f16_config
        const int splits = w4a16::choose_linear_config(M, N, K, w4a16::kMaxKSplits).k_splits;
        wanted = w4a16::linear_workspace_bytes_for(M, N, N < 4096 && K >= 4096 && splits < 2 ? 2 : splits);
    }
    const size_t used = flags & W4A16_FLAG_FORCE_TCGEN05 ? 0 : w4a16_linear_scratch_bytes(M, N, K, w4a16::kGroupFast, flags);
    return used > wanted ? used : wanted;
}

size_t w4a16_linear_workspace_bytes(int64_t M, int64_t N, int64_t K) {
    return w4a16_linear_workspace_bytes_flags(M, N, K, 0);
}

size_t w4a16_linear_scratch_bytes(int64_t M, int64_t N, int64_t K, int64_t group_size, uint32_t flags) {
    if (M <= 0 || N <= 0 || K <= 0 || K % w4a16::kGroupFast != 0 || !w4a16::is_stream_group(group_size)) return 0;
    if (flags & W4A16_FLAG_FORCE_GENERIC) return 0;
    const bool small_group = group_size != w4a16::kGroupFast;
    if (small_group ? small_group_routes_to_gemm(M, flags) : routes_to_tcgen05(M, N, K, flags)) {
        return gemm_on_pairs(M, N, K, SIZE_MAX) ? 0 : w4a16::gemm_scratch_bytes(M, N, K);
    }
    auto streaming = [&](int64_t rows) {
        return w4a16::linear_workspace_bytes_for(
            rows, N, w4a16::choose_linear_config(rows, N, K, w4a16::kMaxKSplits, small_group).k_splits);
    };
    if (!small_group || M <= kSmallGroupRows) return streaming(M);
    const size_t whole = streaming(kSmallGroupRows), rest = M % kSmallGroupRows > 0 ? streaming(M % kSmallGroupRows) : 0;
    return whole > rest ? whole : rest;
}

// w4a16_linear_f16_bias, and w4a16_linear_f16_input without a transform.
static int linear_f16(const void* x, const void* packed, const void* scales, const void* bias, void* y, int64_t M, int64_t N, int64_t K,
                      int64_t group_size, void* workspace, size_t workspace_bytes, uint32_t flags, bool among_transforms,
                      w4a16_stream_t stream) {
    const int status = validate_linear(x, packed, scales, y, M, N, K, group_size);
    if (status != W4A16_OK || M == 0 || N == 0) return status;
    w4a16::LinearProblem p{static_cast<const __half*>(x), static_cast<const uint8_t*>(packed),
                           static_cast<const __half*>(scales), y, M, N, K, group_size,
                           workspace, workspace_bytes};
    p.among_transforms = among_transforms;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const bool out_f32 = (flags & W4A16_FLAG_OUTPUT_F32) != 0;
    p.bias = static_cast<const __half*>(bias);
    if (bias != nullptr && (out_f32 || K == 0)) return W4A16_ERR_BAD_CONFIG;
    if (K == 0) {
        const size_t element = out_f32 ? sizeof(float) : sizeof(__half);
        return cudaMemsetAsync(y, 0, static_cast<size_t>(M) * N * element, s) == cudaSuccess
                   ? W4A16_OK
                   : W4A16_ERR_LAUNCH;
    }
    const bool small_group = small_group_streams(x, packed, scales, K, group_size);
    if ((flags & W4A16_FLAG_FORCE_GENERIC) || (!small_group && !fast_path_applies(x, packed, K, group_size))) {
        return w4a16::launch_linear_generic(p, out_f32, s);
    }
    if (small_group ? small_group_routes_to_gemm(M, flags) : routes_to_tcgen05(M, N, K, flags)) return launch_gemm(p, s);
    if (!small_group || M <= kSmallGroupRows) return launch_streaming(p, small_group, flags, s);
    // Large batches of small groups whose weights may not be rounded: 64 rows after the other, each with the whole workspace to
    // split K into.  (8192 x 8192, 64-wide groups, 65 / 512 rows: 110 / 766 us; the generic kernel 1585 / 11268; the GEMM, with
    // rounded weights, 26 / 68.)
    for (int64_t m = 0; m < M; m += kSmallGroupRows) {
        w4a16::LinearProblem rows = p;
        rows.x += m * K;
        rows.y = static_cast<char*>(p.y) + static_cast<size_t>(m) * N * (out_f32 ? sizeof(float) : sizeof(__half));
        rows.M = M - m < kSmallGroupRows ? M - m : kSmallGroupRows;
        const int launched = launch_streaming(rows, small_group, flags, s);
        if (launched != W4A16_OK) return launched;
    }
    return W4A16_OK;
}

int w4a16_linear_f16(const void* x, const void* packed, const void* scales, void* y, int64_t M, int64_t N,
                     int64_t K, int64_t group_size, void* workspace, size_t workspace_bytes, uint32_t flags,
                     w4a16_stream_t stream) {
    return linear_f16(x, packed, scales, nullptr, y, M, N, K, group_size, workspace, workspace_bytes, flags, false, stream);
}

int w4a16_linear_f16_bias(const void* x, const void* packed, const void* scales, const void* bias, void* y, int64_t M, int64_t N,
                          int64_t K, int64_t group_size, void* workspace, size_t workspace_bytes, uint32_t flags,
                          w4a16_stream_t stream) {
    return linear_f16(x, packed, scales, bias, y, M, N, K, group_size, workspace, workspace_bytes, flags, false, stream);
}

int w4a16_linear_f16_input(const void* x, const void* packed, const void* scales, void* y, int64_t M, int64_t N,
                           int64_t K, int64_t group_size, void* workspace, size_t workspace_bytes, uint32_t flags,
                           const w4a16_input_transform* transform, w4a16_stream_t stream) {
    if (transform == nullptr || transform->kind == W4A16_INPUT_PLAIN) {
        return linear_f16(x, packed, scales, nullptr, y, M, N, K, group_size, workspace, workspace_bytes, flags, true, stream);
    }
    const int status = validate_linear(x, packed, scales, y, M, N, K, group_size);
    if (status != W4A16_OK || M == 0 || N == 0) return status;
    if (K == 0 || M > 64 || !fast_path_applies(x, packed, K, group_size)) return W4A16_ERR_BAD_CONFIG;
    w4a16::LinearProblem p{static_cast<const __half*>(x), static_cast<const uint8_t*>(packed),
                           static_cast<const __half*>(scales), y, M, N, K, group_size,
                           workspace, workspace_bytes, nullptr, transform};
    p.among_transforms = true;
    int max_splits = 1;
    if (workspace != nullptr && aligned16(workspace)) {
        for (int splits = w4a16::kMaxKSplits; splits > 1; splits >>= 1) {
            if (workspace_bytes >= w4a16::linear_workspace_bytes_for(M, N, splits)) {
                max_splits = splits;
                break;
            }
        }
    }
    w4a16_linear_config cfg = w4a16::choose_linear_config(M, N, K, max_splits);
    if (reinterpret_cast<uintptr_t>(scales) % 4 != 0) cfg.unroll = 1;
    return w4a16::launch_linear_mma(p, cfg, (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0,
                                    (flags & W4A16_FLAG_OUTPUT_F32) != 0, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_linear_f16_config(const void* x, const void* packed, const void* scales, void* y, int64_t M,
                            int64_t N, int64_t K, int64_t group_size, void* workspace,
                            size_t workspace_bytes, uint32_t flags, const w4a16_linear_config* config,
                            w4a16_stream_t stream) {
    const int status = validate_linear(x, packed, scales, y, M, N, K, group_size);
    if (status != W4A16_OK || M == 0 || N == 0) return status;
    if (config == nullptr) return W4A16_ERR_NULL_POINTER;
    if (!fast_path_applies(x, packed, K, group_size)) return W4A16_ERR_BAD_CONFIG;
    w4a16_linear_config cfg = w4a16::choose_linear_config(M, N, K, 1);
    if (config->row_tiles) cfg.row_tiles = config->row_tiles;
    if (config->k_warps) cfg.k_warps = config->k_warps;
    if (config->k_splits) cfg.k_splits = config->k_splits;
    if (config->unroll) cfg.unroll = config->unroll;
    if (config->stages) cfg.stages = config->stages;
    w4a16::LinearProblem p{static_cast<const __half*>(x), static_cast<const uint8_t*>(packed),
                           static_cast<const __half*>(scales), y, M, N, K, group_size,
                           workspace, workspace_bytes};
    return w4a16::launch_linear_mma(p, cfg, (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0,
                                    (flags & W4A16_FLAG_OUTPUT_F32) != 0, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_linear_f16_peers(const void* x, int64_t x_ld, const void* packed, const void* scales, void* y, int64_t M,
                           int64_t N, int64_t K, int64_t group_size, void* workspace, size_t workspace_bytes,
                           uint32_t flags, const w4a16_peer_target* target, const w4a16_peer_source* source,
                           w4a16_stream_t stream) {
    // with a target the results go to the ranks' buffers and y is not used
    const int status = validate_linear(x, packed, scales, target != nullptr ? static_cast<const void*>(target) : y, M, N,
                                       K, group_size);
    if (status != W4A16_OK) return status;
    if (M == 0 || N == 0 || K == 0) return W4A16_ERR_BAD_SHAPE;
    if (M > 64 || !fast_path_applies(x, packed, K, group_size)) return W4A16_ERR_BAD_CONFIG;
    w4a16::LinearProblem p{static_cast<const __half*>(x), static_cast<const uint8_t*>(packed),
                           static_cast<const __half*>(scales), target != nullptr ? nullptr : y, M, N, K, group_size,
                           workspace, workspace_bytes, target, nullptr, source, x_ld};
    int max_splits = 1;
    if (workspace != nullptr && aligned16(workspace)) {
        for (int splits = w4a16::kMaxKSplits; splits > 1; splits >>= 1) {
            if (workspace_bytes >= w4a16::linear_workspace_bytes_for(M, N, splits)) {
                max_splits = splits;
                break;
            }
        }
    }
    w4a16_linear_config cfg = w4a16::choose_linear_config(M, N, K, max_splits);
    if (reinterpret_cast<uintptr_t>(scales) % 4 != 0) cfg.unroll = 1;
    return w4a16::launch_linear_mma(p, cfg, (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0,
                                    (flags & W4A16_FLAG_OUTPUT_F32) != 0, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_wait_peers(const w4a16_peer_source* source, const void* buffer0, void* out, int64_t count, uint32_t flags,
                     w4a16_stream_t stream) {
    const int64_t ld = source != nullptr && source->columns_per_rank > 0
                           ? source->columns_per_rank * static_cast<int64_t>(source->world)
                           : 0;
    return w4a16::launch_wait_peers(source, buffer0, out, count, ld, (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0,
                                    reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_sum_partials_f16(const void* partials, void* y, int64_t count, int32_t world, const w4a16_peer_source* source,
                           uint32_t flags, w4a16_stream_t stream) {
    if (count < 0 || world < 1 || world > 32) return W4A16_ERR_BAD_SHAPE;
    if (count == 0) return W4A16_OK;
    if (partials == nullptr || y == nullptr) return W4A16_ERR_NULL_POINTER;
    if (source != nullptr && source->world != world) return W4A16_ERR_BAD_SHAPE;
    return w4a16::launch_sum_partials(partials, static_cast<__half*>(y), count, world, source,
                                      (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_bounds_check_status(uint32_t* site, uint32_t* count) {
    if (site == nullptr || count == nullptr) return W4A16_ERR_NULL_POINTER;
    unsigned s = 0, c = 0;
    const int status = w4a16::read_bounds_check(&s, &c);
    *site = s;
    *count = c;
    return status;
}

int w4a16_device_status(uint32_t* value) {
    if (value == nullptr) return W4A16_ERR_NULL_POINTER;
    unsigned v = 0;
    const int status = w4a16::read_tcgen05_status(&v);
    *value = v;
    return status;
}

int w4a16_dequantize_f16(const void* packed, const void* scales, void* weights, int64_t N, int64_t K,
                         int64_t group_size, w4a16_stream_t stream) {
    if (N < 0 || K < 0 || (K & 1)) return W4A16_ERR_BAD_SHAPE;
    if (group_size <= 0 || group_size % 32 != 0) return W4A16_ERR_BAD_GROUP;
    if (K % group_size != 0) return W4A16_ERR_BAD_SHAPE;
    if (N == 0 || K == 0) return W4A16_OK;
    if (packed == nullptr || scales == nullptr || weights == nullptr) return W4A16_ERR_NULL_POINTER;
    if (!aligned16(packed) || !aligned16(weights)) return W4A16_ERR_MISALIGNED;
    return w4a16::launch_dequantize(static_cast<const uint8_t*>(packed), static_cast<const __half*>(scales),
                                    static_cast<__half*>(weights), N, K, group_size,
                                    reinterpret_cast<cudaStream_t>(stream));
}

static int quantize_pack(const void* weights, bool is_f32, void* packed, void* scales, int64_t N, int64_t K,
                         int64_t group_size, w4a16_stream_t stream) {
    if (N < 0 || K < 0 || (K & 1)) return W4A16_ERR_BAD_SHAPE;
    if (group_size <= 0 || (group_size & 1) || group_size > INT32_MAX) return W4A16_ERR_BAD_GROUP;
    if (K % group_size != 0) return W4A16_ERR_BAD_SHAPE;
    if (N == 0 || K == 0) return W4A16_OK;
    if (weights == nullptr || packed == nullptr || scales == nullptr) return W4A16_ERR_NULL_POINTER;
    if (reinterpret_cast<uintptr_t>(packed) % 2 != 0 || reinterpret_cast<uintptr_t>(scales) % 2 != 0 ||
        reinterpret_cast<uintptr_t>(weights) % (is_f32 ? 4 : 2) != 0) {
        return W4A16_ERR_MISALIGNED;
    }
    return w4a16::launch_quantize_pack(weights, is_f32, static_cast<uint8_t*>(packed), static_cast<__half*>(scales), N, K,
                                       group_size, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_quantize_pack_f16(const void* weights, void* packed, void* scales, int64_t N, int64_t K, int64_t group_size,
                            w4a16_stream_t stream) {
    return quantize_pack(weights, false, packed, scales, N, K, group_size, stream);
}

int w4a16_quantize_pack_f32(const void* weights, void* packed, void* scales, int64_t N, int64_t K, int64_t group_size,
                            w4a16_stream_t stream) {
    return quantize_pack(weights, true, packed, scales, N, K, group_size, stream);
}

int w4a16_add_rmsnorm_f16(const void* stream_in, const void* delta, const void* weight, void* stream_out, void* normed,
                          int64_t hidden, float eps, uint32_t flags, w4a16_stream_t stream) {
    if (hidden <= 0 || hidden > 24576) return W4A16_ERR_BAD_SHAPE;
    if (stream_in == nullptr || weight == nullptr || normed == nullptr) return W4A16_ERR_NULL_POINTER;
    return w4a16::launch_add_rmsnorm(static_cast<const __half*>(stream_in), static_cast<const __half*>(delta),
                                     static_cast<const __half*>(weight), static_cast<__half*>(stream_out),
                                     static_cast<__half*>(normed), static_cast<int>(hidden), eps,
                                     (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_silu_mul_f16(const void* gate_up, void* out, int64_t intermediate, uint32_t flags, w4a16_stream_t stream) {
    if (intermediate <= 0 || intermediate > (1 << 30)) return W4A16_ERR_BAD_SHAPE;
    if (gate_up == nullptr || out == nullptr) return W4A16_ERR_NULL_POINTER;
    return w4a16::launch_silu_mul(static_cast<const __half*>(gate_up), static_cast<__half*>(out),
                                  static_cast<int>(intermediate), (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0,
                                  reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_argmax_advance_f16(const void* logits, int64_t count, int64_t* token, int64_t* position, uint32_t flags,
                             w4a16_stream_t stream) {
    if (count <= 0 || count > INT32_MAX - 8192) return W4A16_ERR_BAD_SHAPE;
    if (logits == nullptr || token == nullptr) return W4A16_ERR_NULL_POINTER;
    return w4a16::launch_argmax_advance(static_cast<const __half*>(logits), static_cast<int>(count),
                                        reinterpret_cast<long long*>(token), reinterpret_cast<long long*>(position),
                                        (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0, reinterpret_cast<cudaStream_t>(stream));
}

size_t w4a16_decode_plan_bytes(const w4a16_decode_model* model) { return w4a16::decode_plan_bytes(model); }

int w4a16_decode_plan_build(const w4a16_decode_model* model, void* plan, size_t plan_bytes, int64_t* token,
                            int64_t* position, w4a16_decode_plan_info* info, w4a16_stream_t stream) {
    return w4a16::decode_plan_build(model, plan, plan_bytes, token, position, info, reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_decode_step_f16(void* plan, const w4a16_decode_plan_info* info, w4a16_stream_t stream) {
    if (plan == nullptr || info == nullptr) return W4A16_ERR_NULL_POINTER;
    return w4a16::launch_decode_step(plan, info->operations, info->grid, info->head_dim, info->smem_bytes,
                                     reinterpret_cast<cudaStream_t>(stream));
}

int w4a16_attention_decode_f16(const void* qkv, void* k_cache, void* v_cache, void* out, const int64_t* position,
                               const float* inv_freq, int32_t q_heads, int32_t kv_heads, int32_t head_dim, int32_t max_len,
                               float rope_scale, float softmax_scale, uint32_t* status, uint32_t flags,
                               w4a16_stream_t stream) {
    if (q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0 || (head_dim != 64 && head_dim != 128) || max_len <= 0) {
        return W4A16_ERR_BAD_SHAPE;
    }
    if (qkv == nullptr || k_cache == nullptr || v_cache == nullptr || out == nullptr || position == nullptr ||
        inv_freq == nullptr || status == nullptr) {
        return W4A16_ERR_NULL_POINTER;
    }
    if (!aligned16(k_cache) || !aligned16(v_cache)) return W4A16_ERR_MISALIGNED;    // rows are read 16 bytes at a time
    return w4a16::launch_attention_decode(static_cast<const __half*>(qkv), static_cast<__half*>(k_cache),
                                          static_cast<__half*>(v_cache), static_cast<__half*>(out),
                                          reinterpret_cast<const long long*>(position), inv_freq, q_heads, kv_heads, head_dim,
                                          max_len, rope_scale, softmax_scale, status,
                                          (flags & W4A16_FLAG_PROGRAMMATIC_LAUNCH) != 0, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
