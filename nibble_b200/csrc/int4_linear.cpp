// Torch operator shim: registers w4a16::linear and w4a16::dequantize for the CUDA dispatch key
// with the schemas of the reference's csrc/int4_linear.cpp:16-28, validates tensors the way its
// int4_linear_cuda / int4_dequantize_cuda do (csrc/int4_linear_kernel.cu:646-691, 809-841: every
// violation is a TORCH_CHECK, i.e. a Python RuntimeError), allocates the output from the caching
// allocator and hands raw pointers plus the current stream to the C ABI in include/w4a16_b200.h.
// No kernel lives here.  linear_module.cpp, the native side of QuantizedLinear.forward, calls these operators.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include <unistd.h>

#include <algorithm>
#include <array>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <optional>
#include <utility>

#include "../../include/w4a16_b200.h"

namespace {

// Scratch of calls that share K between CTAs: arrival counters, zero between calls, and FP32 parts.
constexpr int64_t kWorkspaceBytes = 40 << 20;   // the most: 38 MiB are the GEMM's parts, two of 256 x 128 sums for each of 148 CTAs

// The arrival counters of any problem whose scratch fits: the fixed 256 KB prefix, and then some.
constexpr int64_t kCounterBytes = 1 << 20;

at::Tensor zeroed_scratch(const at::Device& device, cudaStream_t stream, int64_t bytes) {
    at::Tensor scratch = at::detail::empty_cuda({bytes}, at::kByte, device, c10::nullopt);
    C10_CUDA_CHECK(cudaMemsetAsync(scratch.data_ptr(), 0, static_cast<size_t>(std::min(bytes, kCounterBytes)), stream));
    return scratch;
}

// Outside of graph capture: one buffer per (device, stream), so that calls on different streams never share it, allocated and
// zeroed by the first call that needs it and kept, since the kernels leave the counters at zero.  A call that needs more replaces
// it; the caching allocator hands the old one out again on the same stream only, behind the calls that used it.
//
// During capture: memory of the graph's own, zeroed by a node of that graph in front of its first sharing call on the stream.  The
// buffer of the eager calls would tie the graph to counters that another graph or an eager call may not have cleared yet (its
// zeroing would be a node of whichever graph was captured first) or is using at the time of the replay.  It is held until the
// stream's next call outside this capture.  (A zeroing in front of every call costs a replay 3 us each: 28672 -> 8192, one row, 27.8 ->
// 30.8.)
at::Tensor workspace_for(const at::Device& device, cudaStream_t stream, int64_t bytes) {
    struct Kept {
        at::Tensor buffer;
        unsigned long long capture = 0;
    };
    static std::mutex mutex;
    static auto* cache = new std::map<std::pair<int, cudaStream_t>, std::array<Kept, 2>>();   // eager, captured
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    C10_CUDA_CHECK(cudaStreamGetCaptureInfo(stream, &status, &capture));
    const bool capturing = status != cudaStreamCaptureStatusNone;
    std::lock_guard<std::mutex> lock(mutex);
    auto& [eager, captured] = (*cache)[std::make_pair(static_cast<int>(device.index()), stream)];
    if (captured.buffer.defined() && (!capturing || captured.capture != capture)) captured.buffer = at::Tensor();
    Kept& kept = capturing ? captured : eager;
    if (!kept.buffer.defined() || kept.buffer.numel() < bytes) {
        int64_t size = 1 << 20;
        while (size < bytes) size *= 2;
        kept.buffer = at::Tensor();
        kept.buffer = zeroed_scratch(device, stream, std::min(size, kWorkspaceBytes));
        kept.capture = capture;
    }
    return kept.buffer;
}

// The W4A16_* environment variables, read on every call (they may change between calls) in one pass over the environment.
//   W4A16_ROWS_PER_WARP  how many output rows one lane owns: 2 (one 16-row tile per warp) or 4 (two tiles); 1 is accepted
//                        for compatibility and means 2.  Anything else is an error, as in the reference
//                        (csrc/int4_linear_kernel.cu:481-491).
//   W4A16_DECODE         "generic" forces the generic kernel
// (The module heeds the first two as far as heeds_named_kernel says.)
//   W4A16_PDL            "1": weights may be read before the kernel in front has finished
struct EnvironmentChoices {
    int row_tiles = 0;      // 0: not forced
    uint32_t flags = 0;
};
EnvironmentChoices environment_choices() {
    EnvironmentChoices choices;
    for (char** entry = environ; entry != nullptr && *entry != nullptr; ++entry) {
        const char* text = *entry;
        if (text[0] != 'W' || std::strncmp(text, "W4A16_", 6) != 0) continue;
        text += 6;
        if (std::strncmp(text, "ROWS_PER_WARP=", 14) == 0) {
            const int rows = std::atoi(text + 14);
            TORCH_CHECK(rows == 1 || rows == 2 || rows == 4, "W4A16_ROWS_PER_WARP must be 1, 2, or 4");
            choices.row_tiles = rows == 4 ? 2 : 1;
        } else if (std::strcmp(text, "DECODE=generic") == 0) {
            choices.flags |= W4A16_FLAG_FORCE_GENERIC;
        } else if (std::strcmp(text, "PDL=1") == 0) {
            choices.flags |= W4A16_FLAG_PROGRAMMATIC_LAUNCH;
        }
    }
    return choices;
}

void check_status(int status, const char* what) {
    TORCH_CHECK(status == W4A16_OK, what, " failed: ", w4a16_status_string(status));
}

bool aligned16(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }

// Whether the tensor-core kernels take calls of this K and group, and the dequantiser these weights.
bool has_tensor_core_kernel(const at::Tensor& packed_weights, int64_t k, int64_t group_size) {
    return (group_size == 128 || group_size == 64 || group_size == 32) && k > 0 && k % 128 == 0 && aligned16(packed_weights);
}

// Whether such a call has addresses that those kernels do not take: a view at an odd offset, a row slice of a larger scale matrix.
bool declined_for_alignment(const at::Tensor& activations, const at::Tensor& scales, int64_t group_size) {
    return !aligned16(activations) || (group_size != 128 && !aligned16(scales));
}

// Whether a variable of the environment that names a kernel is heeded by the module's call: as far as small and medium batches go,
// which these kernels are for, and one of them refuses larger ones.
bool heeds_named_kernel(int64_t m, int64_t n, int64_t k) {
    if (m <= 256 || n % 8 != 0) return true;
    if (m > 1024 || n > 20 * k) return false;
    return m <= 512 || n * k <= 4 << 20 || (k >= 2048 && m <= 896) || k >= 8 * n;
}

at::Tensor dequantize_cuda_impl(const at::Tensor& packed_weights, const at::Tensor& scales, int64_t group_size);

// The product with dequantised FP16 weights, as the module forms it.  Nothing here takes part in autograd or is cast by autocast:
// the operator's result is FP16 whatever the context.
at::Tensor dequantize_and_multiply(const at::Tensor& activations, const at::Tensor& packed_weights, const at::Tensor& scales,
                                   const at::Tensor* bias, int64_t group_size, int64_t m, at::IntArrayRef shape) {
    const at::AutoDispatchBelowADInplaceOrView below;
    const c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
    const at::Tensor weights = dequantize_cuda_impl(packed_weights, scales, group_size);
    at::Tensor out = at::mm(activations.view({m, weights.size(1)}), weights.t());
    if (bias != nullptr) out.add_(*bias);
    return out.view(shape);
}

// `activations` is [..., K] when `any_rank` (the module's call), else [M, K]; the result keeps its leading dimensions.
at::Tensor linear_impl(const at::Tensor& activations, const at::Tensor& packed_weights, const at::Tensor& scales,
                       const at::Tensor* bias, int64_t group_size, bool out_f32, bool any_rank) {
    TORCH_CHECK(activations.is_cuda(), "activations must be a CUDA tensor");
    TORCH_CHECK(packed_weights.is_cuda(), "packed_weights must be a CUDA tensor");
    TORCH_CHECK(scales.is_cuda(), "scales must be a CUDA tensor");
    TORCH_CHECK(activations.device() == packed_weights.device() && activations.device() == scales.device(),
                "all inputs must be on the same CUDA device");
    TORCH_CHECK(activations.scalar_type() == at::kHalf, "activations must have dtype torch.float16");
    TORCH_CHECK(packed_weights.scalar_type() == at::kByte, "packed_weights must have dtype torch.uint8");
    TORCH_CHECK(scales.scalar_type() == at::kHalf, "scales must have dtype torch.float16");
    if (any_rank) {
        TORCH_CHECK(activations.dim() >= 1, "activations must have shape [..., K]");
    } else {
        TORCH_CHECK(activations.dim() == 2, "activations must have shape [M, K]");
    }
    TORCH_CHECK(packed_weights.dim() == 2, "packed_weights must have shape [N, K / 2]");
    TORCH_CHECK(scales.dim() == 2, "scales must have shape [N, K / group_size]");
    TORCH_CHECK(activations.is_contiguous(), "activations must be contiguous");
    TORCH_CHECK(packed_weights.is_contiguous(), "packed_weights must be contiguous");
    TORCH_CHECK(scales.is_contiguous(), "scales must be contiguous");
    TORCH_CHECK(group_size > 0, "group_size must be greater than zero");
    TORCH_CHECK(group_size % 2 == 0, "group_size must be even because each byte contains two weights");

    const int64_t k = activations.size(-1);
    const int64_t n = packed_weights.size(0);
    TORCH_CHECK(packed_weights.size(1) * 2 == k, "packed_weights and activations must describe the same K dimension");
    TORCH_CHECK(k % group_size == 0, "K must be divisible by group_size");
    TORCH_CHECK(scales.size(0) == n && scales.size(1) == k / group_size,
                "scales must have shape [N, K / group_size]");
    if (bias != nullptr) {
        TORCH_CHECK(bias->device() == activations.device() && bias->scalar_type() == at::kHalf && bias->is_contiguous() &&
                        bias->dim() == 1 && bias->size(0) == n,
                    "bias must be a contiguous float16 tensor with shape [N] on the activations' device");
    }

    const c10::cuda::CUDAGuard guard(activations.device());
    c10::SmallVector<int64_t, 5> shape(activations.sizes().begin(), activations.sizes().end());
    int64_t m = 1;
    for (size_t i = 0; i + 1 < shape.size(); ++i) m *= shape[i];
    shape.back() = n;
    const auto new_output = [&] {
        return at::detail::empty_cuda(shape, out_f32 ? at::kFloat : at::kHalf, activations.device(), c10::nullopt);
    };
    if (m == 0 || n == 0) return new_output();

    const EnvironmentChoices choices = environment_choices();
    // The module's large batches are the product with dequantised FP16 weights whichever kernel forms it, so where the tensor-core
    // kernels decline the addresses this one does: the generic kernel, which takes any, is no match (4096 x 4096, activations at
    // an odd offset, 65 / 777 / 2048 rows: 400 / 4030 / 10460 us with it, 90 / 300 / 640 this way).  The same for batches beyond
    // those that a variable's kernel is meant for (8192 -> 4096, 2048 rows, W4A16_DECODE=generic: 20990 us; W4A16_ROWS_PER_WARP: refused).
    if (any_rank && m > 64 && has_tensor_core_kernel(packed_weights, k, group_size)) {
        const bool generic = (choices.flags & W4A16_FLAG_FORCE_GENERIC) != 0;
        const bool named = generic || (choices.row_tiles != 0 && bias == nullptr && group_size == 128);
        if ((named && !heeds_named_kernel(m, n, k)) || (!generic && declined_for_alignment(activations, scales, group_size))) {
            return dequantize_and_multiply(activations, packed_weights, scales, bias, group_size, m, shape);
        }
    }
    at::Tensor output = new_output();
    const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
    // (the module's large batches are the product with dequantised FP16 weights, whichever kernel forms it)
    const uint32_t flags = choices.flags | (out_f32 ? W4A16_FLAG_OUTPUT_F32 : 0u) | (any_rank ? W4A16_FLAG_FP16_WEIGHTS : 0u);
    const int forced_tiles = choices.row_tiles;

    at::Tensor scratch;      // held until the call is enqueued, whatever other threads do with the stream's buffer
    void* workspace = nullptr;
    size_t workspace_bytes = 0;
    const size_t wanted = w4a16_linear_scratch_bytes(m, n, k, group_size, flags);
    if (wanted > 0) {
        scratch = workspace_for(activations.device(), stream, std::min<int64_t>(static_cast<int64_t>(wanted), kWorkspaceBytes));
        workspace = scratch.data_ptr();
        workspace_bytes = static_cast<size_t>(scratch.numel());
    }

    int status;
    if (forced_tiles != 0 && bias == nullptr && !(flags & W4A16_FLAG_FORCE_GENERIC) && group_size == 128 &&
        reinterpret_cast<uintptr_t>(activations.data_ptr()) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(packed_weights.data_ptr()) % 16 == 0) {
        w4a16_linear_config config = {forced_tiles, 0, 0, 0, 0};
        status = w4a16_linear_f16_config(activations.data_ptr(), packed_weights.data_ptr(), scales.data_ptr(),
                                         output.data_ptr(), m, n, k, group_size, workspace, workspace_bytes,
                                         flags, &config, reinterpret_cast<w4a16_stream_t>(stream));
    } else {
        // (an empty K leaves zeros, which the C entry point does not add a bias to)
        const bool fold = bias != nullptr && k > 0;
        status = w4a16_linear_f16_bias(activations.data_ptr(), packed_weights.data_ptr(), scales.data_ptr(),
                                       fold ? bias->data_ptr() : nullptr, output.data_ptr(), m, n, k, group_size, workspace,
                                       workspace_bytes, flags, reinterpret_cast<w4a16_stream_t>(stream));
        if (bias != nullptr && !fold) output.add_(*bias);
    }
    check_status(status, "w4a16::linear");
    return output;
}

at::Tensor linear_cuda_impl(const at::Tensor& activations, const at::Tensor& packed_weights,
                            const at::Tensor& scales, int64_t group_size) {
    return linear_impl(activations, packed_weights, scales, nullptr, group_size, false, false);
}

// Same product with the unrounded FP32 sums as output: the per-device partial of a K-sharded layer.
at::Tensor linear_partial_cuda_impl(const at::Tensor& activations, const at::Tensor& packed_weights,
                                    const at::Tensor& scales, int64_t group_size) {
    return linear_impl(activations, packed_weights, scales, nullptr, group_size, true, false);
}

// The module's whole fused call: activations of any rank, and the bias inside the kernel.
at::Tensor linear_bias_cuda_impl(const at::Tensor& activations, const at::Tensor& packed_weights, const at::Tensor& scales,
                                 const std::optional<at::Tensor>& bias, int64_t group_size) {
    return linear_impl(activations, packed_weights, scales, bias.has_value() ? &*bias : nullptr, group_size, false, true);
}

at::Tensor dequantize_cuda_impl(const at::Tensor& packed_weights, const at::Tensor& scales, int64_t group_size) {
    TORCH_CHECK(packed_weights.is_cuda(), "packed_weights must be a CUDA tensor");
    TORCH_CHECK(scales.is_cuda(), "scales must be a CUDA tensor");
    TORCH_CHECK(packed_weights.device() == scales.device(),
                "packed_weights and scales must be on the same CUDA device");
    TORCH_CHECK(packed_weights.scalar_type() == at::kByte, "packed_weights must have dtype torch.uint8");
    TORCH_CHECK(scales.scalar_type() == at::kHalf, "scales must have dtype torch.float16");
    TORCH_CHECK(packed_weights.dim() == 2, "packed_weights must have shape [N, K / 2]");
    TORCH_CHECK(scales.dim() == 2, "scales must have shape [N, K / group_size]");
    TORCH_CHECK(packed_weights.is_contiguous(), "packed_weights must be contiguous");
    TORCH_CHECK(scales.is_contiguous(), "scales must be contiguous");
    TORCH_CHECK(group_size > 0 && group_size % 32 == 0,
                "dequantize needs group_size to be a positive multiple of 32");
    TORCH_CHECK(reinterpret_cast<uintptr_t>(packed_weights.data_ptr()) % 16 == 0,
                "packed_weights must be 16-byte aligned");

    const int64_t n = packed_weights.size(0);
    const int64_t k = packed_weights.size(1) * 2;
    TORCH_CHECK(k % group_size == 0, "K must be divisible by group_size");
    TORCH_CHECK(scales.size(0) == n && scales.size(1) == k / group_size,
                "scales must have shape [N, K / group_size]");

    const c10::cuda::CUDAGuard guard(packed_weights.device());
    at::Tensor weights = at::empty({n, k}, packed_weights.options().dtype(at::kHalf));
    if (n == 0 || k == 0) return weights;
    const int status = w4a16_dequantize_f16(
        packed_weights.data_ptr(), scales.data_ptr(), weights.data_ptr(), n, k, group_size,
        reinterpret_cast<w4a16_stream_t>(at::cuda::getCurrentCUDAStream().stream()));
    check_status(status, "w4a16::dequantize");
    return weights;
}

std::tuple<at::Tensor, at::Tensor> quantize_pack_cuda_impl(const at::Tensor& weights, int64_t group_size) {
    TORCH_CHECK(weights.is_cuda(), "weights must be a CUDA tensor");
    TORCH_CHECK(weights.scalar_type() == at::kHalf || weights.scalar_type() == at::kFloat,
                "weights must have dtype torch.float16 or torch.float32");
    TORCH_CHECK(weights.dim() == 2, "weights must have shape [N, K]");
    TORCH_CHECK(group_size > 0, "group_size must be greater than zero");
    TORCH_CHECK(weights.size(1) % group_size == 0, "K must be divisible by group_size");
    TORCH_CHECK(weights.size(1) % 2 == 0 && group_size % 2 == 0, "K and group_size must be even: one byte carries two weights");
    const at::Tensor dense = weights.contiguous();
    const int64_t n = dense.size(0);
    const int64_t k = dense.size(1);
    const c10::cuda::CUDAGuard guard(dense.device());
    at::Tensor packed = at::empty({n, k / 2}, dense.options().dtype(at::kByte));
    at::Tensor scales = at::empty({n, k / group_size}, dense.options().dtype(at::kHalf));
    if (n == 0 || k == 0) return {packed, scales};
    const auto stream = reinterpret_cast<w4a16_stream_t>(at::cuda::getCurrentCUDAStream().stream());
    const int status = dense.scalar_type() == at::kFloat
                           ? w4a16_quantize_pack_f32(dense.data_ptr(), packed.data_ptr(), scales.data_ptr(), n, k, group_size, stream)
                           : w4a16_quantize_pack_f16(dense.data_ptr(), packed.data_ptr(), scales.data_ptr(), n, k, group_size, stream);
    check_status(status, "w4a16::quantize_pack");
    return {packed, scales};
}

}  // namespace

TORCH_LIBRARY(w4a16, m) {
    m.def("linear(Tensor activations, Tensor packed_weights, Tensor scales, int group_size) -> Tensor");
    // not in the reference: any rank, bias added in the kernel
    m.def("linear_bias(Tensor activations, Tensor packed_weights, Tensor scales, Tensor? bias, int group_size) -> Tensor");
    m.def("dequantize(Tensor packed_weights, Tensor scales, int group_size) -> Tensor");
    // not in the reference: FP32 partial sums for layers sharded along K
    m.def("linear_partial(Tensor activations, Tensor packed_weights, Tensor scales, int group_size) -> Tensor");
    // not in the reference: its quantiser is host code (w4a16/quantization.py:65-113)
    m.def("quantize_pack(Tensor weights, int group_size) -> (Tensor, Tensor)");
}

TORCH_LIBRARY_IMPL(w4a16, CUDA, m) {
    m.impl("linear", &linear_cuda_impl);
    m.impl("linear_bias", &linear_bias_cuda_impl);
    m.impl("dequantize", &dequantize_cuda_impl);
    m.impl("linear_partial", &linear_partial_cuda_impl);
    m.impl("quantize_pack", &quantize_pack_cuda_impl);
}
