// The Python entry points' native side: QuantizedLinear.forward in one call, and the operators without torch.ops.
//
// The module's Python forward checks its arguments, flattens them, goes through torch.ops and reshapes: about 8 us of
// interpreter and binding time around a 2 us kernel at M = 1.  linear_forward() makes the same checks and calls the same
// operators through their dispatcher handles (so profilers, dispatch modes and fake tensors see them as before) in a
// quarter of that.  It takes only the ordinary case -- a plain, contiguous FP16 CUDA tensor outside tracing, autocast and
// function modes -- and returns NotImplemented for everything else, including every invalid call: the Python code then
// decides, and raises what it always raised.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/core/InferenceMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <algorithm>
#include <optional>
#include <tuple>

namespace {

using QuantizePack = std::tuple<at::Tensor, at::Tensor>(const at::Tensor&, int64_t);
using Linear = at::Tensor(const at::Tensor&, const at::Tensor&, const at::Tensor&, int64_t);
using LinearBias = at::Tensor(const at::Tensor&, const at::Tensor&, const at::Tensor&, const std::optional<at::Tensor>&, int64_t);
using Dequantize = at::Tensor(const at::Tensor&, const at::Tensor&, int64_t);

template <typename Signature>
c10::TypedOperatorHandle<Signature> operator_handle(const char* name) {
    return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Signature>();
}

// Whether the operator is the faster way for 897 to 4096 rows, by models of both (us).  Their constants are fitted to the times of both
// on 259 calls on layers of 512 to 28416 -> 256 to 20992, in runs of 14 ms.  On 700 other calls (by which the term for few tiles was
// set) choosing by them is 0.8 % slower than the better way on average, and more than 3 % slower than the product on 24.  By the depth
// of the layer alone (K >= 2048 to the operator) it was 2.1 % and 142, and narrow layers, which leave half of the SMs without a tile,
// took up to 1.6 times as long (7296 -> 384, 3072 rows: 31 / 20; 8192 -> 1024, 1536 rows: 33 / 27).
bool operator_is_faster(int64_t rows, int64_t out_features, int64_t in_features) {
    const int64_t k_blocks = in_features / 128, n_tiles = (out_features + 255) / 256;
    const int64_t tiles = n_tiles * ((rows + 127) / 128), pair_tiles = n_tiles * ((rows + 255) / 256);
    // whole rounds of pairs of SMs; or clusters of up to eight SMs that share a tile, or all SMs in equal runs
    double by_operator = 2.5 + static_cast<double>((pair_tiles + 73) / 74) * (2.0 + 0.84 * static_cast<double>(k_blocks));
    double single = by_operator;
    if (tiles <= 148) {
        const int64_t sharing = tiles > 74 ? 1 : tiles > 44 ? 2 : std::min<int64_t>(8, 132 / tiles);
        single = (sharing > 1 ? 10.0 : 6.5) + 0.8 * static_cast<double>((k_blocks + sharing - 1) / sharing);
    } else if ((tiles <= 296 && in_features >= 4096) || (rows <= 1024 && in_features >= 2048)) {
        single = 20.0 + static_cast<double>(tiles * k_blocks) / 148.0;
    }
    if (single < by_operator) by_operator = single;
    const double weights = static_cast<double>(out_features) * static_cast<double>(in_features);
    double by_product = 7.0 + weights / 1.75e6 + static_cast<double>(rows) * weights / 6.1e8;
    if (tiles <= 33) by_product += 0.04 * static_cast<double>(k_blocks);      // cuBLAS is short of tiles too (17792 -> 256, 1792 rows: 24 / 33)
    return by_operator < (by_product > 15.5 ? by_product : 15.5);      // (two launches and their operators: 15.5 us of host time)
}

// Whether a batch goes to the fused operator, or is multiplied by dequantised FP16 weights (same arithmetic from 65 rows
// on: weights rounded to FP16, FP32 sums).  linear.py states the same rule (takes_operator) for the calls that stay in Python; a
// test holds the two together.  The lines come from times of both on 34 layers from 512 x 1024 to 28672 x 8192 at 160 to 8192 rows,
// back to back for 12 ms and more, so that the clocks are those of a long run (us, the operator / dequantise and multiply):
//   - cuBLAS falls off its fast kernels where an output row is no multiple of 16 bytes (9216 -> 2575, 128 rows: 20 / 125);
//   - up to 512 rows the operator, never slower (8192 -> 28672, 512 rows: 201 / 374);
//   - 513 to 896 rows: all but shallow layers (8320 -> 6400, 702 rows: 65 / 85; 512 -> 28672, 777 rows: 1.16 times as long);
//   - to 1024 rows: of those the small or narrow ones (3456 -> 256, 1024 rows: 13.8 / 15.6), and else
//   - to 4096 rows: where the models above say so (8192 -> 28672, 2048 rows: 730 to 740 / 930 to 990);
//   - above, the weights' round trip costs little beside the product (16384 rows: level, 0.88 to 1.09 times as long).  At 5000 and 8192
//     rows layers with K and N >= 4096 would gain (8192 -> 28672: 0.94 and 0.96 times as long), shallower ones lose up to 5 %.
bool uses_fused_kernel(int64_t rows, int64_t out_features, int64_t in_features, int64_t group_size) {
    if (rows <= 64) return true;
    if (group_size % 32 != 0) return true;
    if ((group_size != 128 && group_size != 64 && group_size != 32) || in_features % 128 != 0) {
        return false;      // the operator has no tensor-core kernel for these (3072 -> 4096 in groups of 96, 65 / 2048 rows: 294 / 7917 us)
    }
    if (out_features % 8 != 0 || rows <= 512) return true;
    if (rows <= 1024) {
        if (out_features > 20 * in_features) return false;
        if (rows <= 896 || out_features * in_features <= 4 << 20 || in_features >= 8 * out_features) return true;
        return operator_is_faster(rows, out_features, in_features);
    }
    if (rows > 4096 || (in_features < 2048 && (out_features + 255) / 256 * ((rows + 127) / 128) > 148)) return false;
    return operator_is_faster(rows, out_features, in_features);
}

// A tensor nobody has subclassed, wrapped or asked to track gradients of.
bool plain(PyObject* object) {
    if (!THPVariable_CheckExact(object)) return false;
    const at::Tensor& t = THPVariable_Unpack(object);
    return t.is_cuda() && !t.requires_grad() && t.is_contiguous() &&
           !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                                     c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched}));
}

// Nothing that wants to see or change calls made from Python is active.
bool ordinary_context() {
    return !at::impl::torch_function_mode_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
           !torch::jit::tracer::isTracing() && !at::autocast::is_autocast_enabled(at::kCUDA);
}

// linear(activations, packed_weights, scales, group_size) -> Tensor or NotImplemented
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 4 || !plain(args[0]) || !plain(args[1]) || !plain(args[2]) || !PyLong_Check(args[3]) || !ordinary_context()) {
        Py_RETURN_NOTIMPLEMENTED;
    }
    const int64_t group_size = PyLong_AsLongLong(args[3]);
    if (PyErr_Occurred() != nullptr) return nullptr;
    at::Tensor out;
    {
        pybind11::gil_scoped_release unlocked;
        const at::AutoDispatchBelowADInplaceOrView below;
        static const auto op = operator_handle<Linear>("w4a16::linear");
        out = op.call(THPVariable_Unpack(args[0]), THPVariable_Unpack(args[1]), THPVariable_Unpack(args[2]), group_size);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// dequantize(packed_weights, scales, group_size) -> Tensor or NotImplemented
PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 3 || !plain(args[0]) || !plain(args[1]) || !PyLong_Check(args[2]) || !ordinary_context()) Py_RETURN_NOTIMPLEMENTED;
    const int64_t group_size = PyLong_AsLongLong(args[2]);
    if (PyErr_Occurred() != nullptr) return nullptr;
    at::Tensor out;
    {
        pybind11::gil_scoped_release unlocked;
        const at::AutoDispatchBelowADInplaceOrView below;
        static const auto op = operator_handle<Dequantize>("w4a16::dequantize");
        out = op.call(THPVariable_Unpack(args[0]), THPVariable_Unpack(args[1]), group_size);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// quantize_pack(weights, group_size) -> (packed, scales) or NotImplemented
PyObject* quantize_pack(PyObject*, PyObject* const* args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 2 || !plain(args[0]) || !PyLong_Check(args[1]) || !ordinary_context()) Py_RETURN_NOTIMPLEMENTED;
    const int64_t group_size = PyLong_AsLongLong(args[1]);
    if (PyErr_Occurred() != nullptr) return nullptr;
    std::tuple<at::Tensor, at::Tensor> out;
    {
        pybind11::gil_scoped_release unlocked;
        const at::AutoDispatchBelowADInplaceOrView below;
        static const auto op = operator_handle<QuantizePack>("w4a16::quantize_pack");
        out = op.call(THPVariable_Unpack(args[0]), group_size);
    }
    PyObject* packed = THPVariable_Wrap(std::move(std::get<0>(out)));
    PyObject* scales = packed == nullptr ? nullptr : THPVariable_Wrap(std::move(std::get<1>(out)));
    PyObject* pair = scales == nullptr ? nullptr : PyTuple_Pack(2, packed, scales);
    Py_XDECREF(packed);
    Py_XDECREF(scales);
    return pair;
    END_HANDLE_TH_ERRORS
}

// linear_forward(activations, packed_weights, scales, bias or None, group_size, fused) -> Tensor or NotImplemented
PyObject* linear_forward(PyObject*, PyObject* const* args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != 6 || !plain(args[0]) || !plain(args[1]) || !plain(args[2]) || (args[3] != Py_None && !plain(args[3])) ||
        !ordinary_context()) {
        Py_RETURN_NOTIMPLEMENTED;
    }
    const at::Tensor& x = THPVariable_Unpack(args[0]);
    // forward-mode differentiation follows the product with dequantised weights (of the activations alone: asked of the buffers,
    // which are views, it takes 0.1 us)
    if (x._fw_grad(/*level=*/0).defined()) Py_RETURN_NOTIMPLEMENTED;
    const at::Tensor& packed = THPVariable_Unpack(args[1]);
    const at::Tensor& scales = THPVariable_Unpack(args[2]);
    std::optional<at::Tensor> bias;
    if (args[3] != Py_None) bias = THPVariable_Unpack(args[3]);
    const int64_t group_size = PyLong_AsLongLong(args[4]);
    const int fused = PyObject_IsTrue(args[5]);
    if (PyErr_Occurred() != nullptr) return nullptr;
    if (x.dim() < 1 || x.scalar_type() != at::kHalf || packed.dim() != 2 || x.size(-1) != packed.size(1) * 2 || x.size(-1) == 0 ||
        group_size <= 0 || x.device() != packed.device() || x.device() != scales.device()) {
        Py_RETURN_NOTIMPLEMENTED;
    }
    const int64_t rows = x.numel() / x.size(-1);
    at::Tensor out;
    {
        pybind11::gil_scoped_release unlocked;             // a launch may block when the stream's queue is full
        const at::AutoDispatchBelowADInplaceOrView below;  // nothing here takes part in autograd
        if ((fused != 0 || group_size % 32 != 0) && uses_fused_kernel(rows, packed.size(0), x.size(-1), group_size)) {
            static const auto op = operator_handle<LinearBias>("w4a16::linear_bias");
            out = op.call(x, packed, scales, bias, group_size);
        } else {
            static const auto op = operator_handle<Dequantize>("w4a16::dequantize");
            // (at::mm on two dimensions rather than at::linear, which takes 2 us longer to get there)
            const at::Tensor weights = op.call(packed, scales, group_size);
            out = at::mm(x.view({rows, x.size(-1)}), weights.t());
            if (bias.has_value()) out.add_(*bias);
            if (x.dim() != 2) {
                c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
                shape.back() = weights.size(0);
                out = out.view(shape);
            }
        }
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// uses_fused_kernel(rows, out_features, in_features, group_size) -> bool
PyObject* rule(PyObject*, PyObject* const* args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    int64_t value[4] = {};
    if (count != 4) {
        PyErr_SetString(PyExc_TypeError, "uses_fused_kernel takes four integers");
        return nullptr;
    }
    for (int i = 0; i < 4; ++i) {
        value[i] = PyLong_AsLongLong(args[i]);
        if (PyErr_Occurred() != nullptr) return nullptr;
    }
    if (uses_fused_kernel(value[0], value[1], value[2], value[3])) Py_RETURN_TRUE;
    Py_RETURN_FALSE;
    END_HANDLE_TH_ERRORS
}

using FastCall = PyObject* (*)(PyObject*, PyObject* const*, Py_ssize_t);
PyCFunction method(FastCall f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {
    {"linear_forward", method(linear_forward), METH_FASTCALL,
     "linear_forward(activations, packed_weights, scales, bias, group_size, fused) -> Tensor or NotImplemented"},
    {"linear", method(linear), METH_FASTCALL, "linear(activations, packed_weights, scales, group_size) -> Tensor or NotImplemented"},
    {"dequantize", method(dequantize), METH_FASTCALL, "dequantize(packed_weights, scales, group_size) -> Tensor or NotImplemented"},
    {"quantize_pack", method(quantize_pack), METH_FASTCALL, "quantize_pack(weights, group_size) -> (Tensor, Tensor) or NotImplemented"},
    {"uses_fused_kernel", method(rule), METH_FASTCALL, "uses_fused_kernel(rows, out_features, in_features, group_size) -> bool"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_C", "Native side of nibble_b200: torch operators and QuantizedLinear.forward.", -1,
                          methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__C() { return PyModule_Create(&module_def); }
