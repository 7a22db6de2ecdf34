"""-m gpu: QuantizedLinear and the model-surgery helpers on a CUDA device
(reference tests/test_linear.py:130-243, tests/test_integration.py:157-204, tests/test_cuda.py:535-556)."""
from __future__ import annotations

import numpy as np
import pytest
import torch
import torch.nn.functional as F

from capi_helpers import check_against_oracle
from nibble_b200 import QuantizedLinear, load_packed_state_dict, quantize_and_pack_weights, replace_linear_layers
from nibble_b200.linear import FUSED_MAX_ROWS
from oracle import w4a16_oracle as oracle

pytestmark = pytest.mark.gpu


def _layer(n=8, k=128, bias=False, fused=True, seed=0):
    torch.manual_seed(seed)
    w = torch.randn((n, k), dtype=torch.float16, device="cuda")
    packed, scales = quantize_and_pack_weights(w, 128)
    b = torch.randn((n,), dtype=torch.float16, device="cuda") if bias else None
    return QuantizedLinear(packed, scales, 128, bias=b, fused=fused)


def _oracle_out(layer, x):
    y = oracle.linear_reference(x.reshape(-1, layer.in_features).cpu().numpy(), layer.packed_weights.cpu().numpy(),
                                layer.scales.cpu().numpy(), layer.group_size)
    y = torch.from_numpy(y).reshape(*x.shape[:-1], layer.out_features)
    return y if layer.bias is None else y + layer.bias.cpu()


@pytest.mark.parametrize("rows", [1, 2, 16])
def test_module_matches_oracle_with_bias(rows):
    layer = _layer(bias=True)
    x = torch.randn((rows, 128), dtype=torch.float16, device="cuda")
    torch.testing.assert_close(layer(x).cpu(), _oracle_out(layer, x), rtol=1e-2, atol=1e-2)


def test_module_accepts_noncontiguous_and_3d():
    layer = _layer()
    x = torch.randn((2, 3, 256), dtype=torch.float16, device="cuda")[..., :128]
    assert not x.is_contiguous()
    out = layer(x)
    assert out.shape == (2, 3, 8)
    torch.testing.assert_close(out.cpu(), _oracle_out(layer, x.contiguous()), rtol=1e-2, atol=1e-2)


def test_large_batch_and_unfused_mode_match_fp16_matmul_of_dequantised_weights():
    layer = _layer(n=64, k=512, seed=2)
    w16 = torch.from_numpy(
        oracle.dequantize_weights(layer.packed_weights.cpu().numpy(), layer.scales.cpu().numpy(), 128).astype(np.float16)
    ).cuda()
    big = torch.randn((FUSED_MAX_ROWS + 5, 512), dtype=torch.float16, device="cuda")
    torch.testing.assert_close(layer(big), F.linear(big, w16), rtol=1e-3, atol=1e-3)
    layer.fused = False
    one = torch.randn((1, 512), dtype=torch.float16, device="cuda")
    torch.testing.assert_close(layer(one), F.linear(one, w16), rtol=1e-3, atol=1e-3)


def test_prefill_batch_on_a_wide_layer_takes_the_tensor_core_kernel():
    from nibble_b200 import _native
    from nibble_b200.linear import PREFILL_MIN_WEIGHT_TILES, uses_fused_kernel

    n = 128 * PREFILL_MIN_WEIGHT_TILES
    layer = _layer(n=n, k=1024, seed=3)
    w16 = torch.from_numpy(
        oracle.dequantize_weights(layer.packed_weights.cpu().numpy(), layer.scales.cpu().numpy(), 128).astype(np.float16)
    ).cuda()
    x = torch.randn((3, 100, 1024), dtype=torch.float16, device="cuda")
    assert uses_fused_kernel(300, n, 128)
    before = _native.core().w4a16_launch_count()
    out = layer(x)
    assert _native.core().w4a16_launch_count() == before + 1      # one fused launch, no dequantise pass
    torch.testing.assert_close(out, F.linear(x, w16), rtol=2e-3, atol=2e-3)


def test_replace_linear_layers_on_cuda_model():
    torch.manual_seed(1)
    model = torch.nn.Sequential(
        torch.nn.Linear(256, 512, bias=True), torch.nn.SiLU(), torch.nn.Linear(512, 128, bias=False)
    ).half().cuda()
    x = torch.randn((4, 256), dtype=torch.float16, device="cuda")
    assert replace_linear_layers(model, group_size=128) == 2
    first = model[0]
    check_against_oracle(first(x) - first.bias, x, first.packed_weights, first.scales)
    assert model(x).shape == (4, 128)


def test_packed_load_never_materialises_fp16_weights():
    n = k = 2048
    source = torch.nn.Linear(k, n, bias=False, dtype=torch.float16)
    q = QuantizedLinear.from_float(source, group_size=128)
    state = {"layer.packed_weights": q.packed_weights.clone(), "layer.scales": q.scales.clone()}

    class Wrapper(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.layer = torch.nn.Linear(k, n, bias=False, dtype=torch.float16)

    with torch.device("meta"):
        model = Wrapper()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    assert load_packed_state_dict(model, state, group_size=128, device="cuda") == 1
    delta = torch.cuda.memory_allocated() - before
    packed_bytes = q.packed_weights.numel() + 2 * q.scales.numel()
    assert model.layer.packed_weights.is_cuda
    assert packed_bytes <= delta < 2 * n * k
    x = torch.randn((1, k), dtype=torch.float16, device="cuda")
    check_against_oracle(model.layer(x), x, model.layer.packed_weights, model.layer.scales)


@pytest.mark.parametrize("rows", [1, 4, 24])
def test_traces_under_torch_compile_aot_eager(rows):
    layer = _layer(n=16, k=256, seed=3)
    x = torch.randn((rows, 256), dtype=torch.float16, device="cuda")
    compiled = torch.compile(layer, backend="aot_eager", fullgraph=True)
    assert torch.equal(compiled(x), layer(x))


def test_fused_siblings_one_launch_same_numbers():
    from nibble_b200 import _native, fuse_parallel_linears

    class Attn(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.q_proj = torch.nn.Linear(2048, 2048, bias=False)
            self.k_proj = torch.nn.Linear(2048, 256, bias=False)
            self.v_proj = torch.nn.Linear(2048, 256, bias=False)

        def forward(self, x):
            return self.q_proj(x), self.k_proj(x), self.v_proj(x)

    torch.manual_seed(4)
    attn = Attn().half().cuda()
    assert replace_linear_layers(attn, group_size=128, fuse_siblings=False) == 3
    x = torch.randn((1, 1, 2048), dtype=torch.float16, device="cuda")
    separate = [t.clone() for t in attn(x)]
    packed = [m.packed_weights.clone() for m in (attn.q_proj, attn.k_proj, attn.v_proj)]
    scales = [m.scales.clone() for m in (attn.q_proj, attn.k_proj, attn.v_proj)]
    assert fuse_parallel_linears(attn) == 1
    before = _native.core().w4a16_launch_count()
    fused = attn(x)
    assert _native.core().w4a16_launch_count() == before + 1
    for got, ref, p, s in zip(fused, separate, packed, scales):
        assert got.shape == ref.shape
        torch.testing.assert_close(got, ref, rtol=1e-2, atol=1e-2)
        check_against_oracle(got.reshape(1, -1), x.reshape(1, -1), p, s)


def test_model_checkpoint_loads_straight_onto_the_device(tmp_path):
    """A file in the reference's model-checkpoint format (scripts/generate.py:214-257) into a meta-device model:
    packed tensors go straight to the GPU, FP16 linear weights never exist, the block computes what the source
    block computes."""
    from nibble_b200 import load_packed_model, save_quantized_model_checkpoint
    from test_fusion_host_logic import Block

    torch.manual_seed(6)
    source = Block(hidden=1024, kv=256, inter=2048, bias=True).half()
    assert replace_linear_layers(source, group_size=128) == 7        # quantised on the host
    path = tmp_path / "model.pt"
    save_quantized_model_checkpoint(path, source, group_size=128, source_model="gpu-test")
    with torch.device("meta"):
        target = Block(hidden=1024, kv=256, inter=2048, bias=True).half()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    assert load_packed_model(target, path, device="cuda") == 7
    delta = torch.cuda.memory_allocated() - before
    packed_bytes = sum(t.numel() * t.element_size() for t in source.state_dict().values())
    fp16_bytes = 2 * sum(m.in_features * m.out_features for m in source.modules() if isinstance(m, QuantizedLinear))
    assert packed_bytes <= delta < fp16_bytes / 2
    for key, tensor in source.state_dict().items():
        got = target.state_dict()[key]
        assert got.is_cuda and torch.equal(got.cpu(), tensor), key
    x = torch.randn((2, 1024), dtype=torch.float16, device="cuda")
    q = target.q_proj
    check_against_oracle(q(x) - q.bias, x, q.packed_weights, q.scales)
    assert target(x).shape == (2, 1024) and not torch.isnan(target(x)).any()


@pytest.mark.parametrize(("k", "n"), [(1024, 77), (8192, 1024), (4096, 5248)])
@pytest.mark.parametrize("rows", [1, 7, 13, 48, 100, 300])
def test_native_forward_equals_the_python_forward(rows, k, n):
    """The native call (bias added inside the kernel) against the operators plus a separate addition, for streaming, split
    and GEMM launches, with any leading dimensions.  Same bits where both take the same kernel."""
    from nibble_b200 import linear as linear_module

    g = torch.Generator().manual_seed(rows + n)
    packed, scales = quantize_and_pack_weights((torch.randn((n, k), generator=g) * 0.02).cuda(), 128)
    x = torch.randn((1, rows, k), generator=g).half().cuda()
    for bias in (None, torch.randn((n,), generator=g).half().cuda()):
        layer = QuantizedLinear(packed, scales, 128, bias=bias)
        native = linear_module.linear_forward(x, packed, scales, bias, 128, True)
        assert native is not NotImplemented and native.shape == (1, rows, n)
        use_fused = linear_module.uses_fused_kernel(rows, n, 128)
        run = linear_module._run_fused if use_fused else linear_module._run_dequant_matmul
        want = run(x.view(rows, k), packed, scales, 128).view(1, rows, n)
        biased = want if bias is None else want + bias
        assert torch.equal(native, biased) if rows <= 64 else torch.allclose(native, biased, rtol=2e-3, atol=2e-3)
        assert torch.equal(layer(x), native)
    # what the native call does not take, the module still does
    wide = torch.zeros((rows + 1, 2 * k), dtype=torch.float16, device="cuda")[:rows]
    wide[:, :k] = x[0]
    assert rows == 1 or linear_module.linear_forward(wide[:, :k], packed, scales, None, 128, True) is NotImplemented
    torch.testing.assert_close(QuantizedLinear(packed, scales, 128)(wide[:, :k]), want[0], rtol=2e-3, atol=2e-3)


class _Passing(torch.overrides.TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize(("n", "k", "gs"), [(1000, 1152, 128), (2048, 5632, 128), (520, 1024, 64), (5003, 512, 32), (8192, 512, 128)])
@pytest.mark.parametrize("rows", [1, 48, 65, 130, 300, 600, 777, 1024, 1100])
def test_every_way_into_the_module_takes_the_native_route(rows, n, k, gs):
    """Autocast, a function mode, non-contiguous activations and compiled code: the bits and the launches of the plain call."""
    from nibble_b200 import _native

    count = _native.core().w4a16_launch_count
    torch.manual_seed(rows + n)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    scales = (torch.rand((n, k // gs), device="cuda") * 0.01 + 1e-3).half()
    x = torch.randn((rows, k), device="cuda").half()
    spaced = torch.zeros((rows, 2 * k), dtype=torch.float16, device="cuda")[:, :k].copy_(x)
    for bias in (None, torch.randn((n,), device="cuda").half()):
        layer = QuantizedLinear(packed, scales, gs, bias=bias)
        before = count()
        want = layer(x)
        launches = count() - before
        w16 = torch.ops.w4a16.dequantize(packed, scales, gs).float()
        exact = x.float() @ w16.t() + (0 if bias is None else bias.float())
        torch.testing.assert_close(want.float(), exact, rtol=2e-3, atol=2e-2)
        before = count()
        with _Passing():
            assert torch.equal(layer(x), want)
        with torch.autocast("cuda", dtype=torch.float16):
            assert torch.equal(layer(x), want)
        if rows > 1:
            assert not spaced.is_contiguous() and torch.equal(layer(spaced), want)
        assert count() - before == (3 if rows > 1 else 2) * launches
    torch._dynamo.reset()
    assert torch.equal(torch.compile(layer, backend="aot_eager", fullgraph=True, dynamic=False)(x), want)


@pytest.mark.parametrize(("k", "n"), [(1024, 264), (2048, 77)])
@pytest.mark.parametrize("gs", [128, 64])
@pytest.mark.parametrize("rows", [65, 777, 2048])
def test_large_batches_at_odd_addresses_are_the_product_with_dequantised_weights(rows, gs, k, n):
    """Activations, or scales of 64-wide groups, that the tensor-core kernels decline for their alignment: the dequantiser and a
    matrix product, with its very bits, whichever way the call comes in; no generic kernel, which takes up to sixteen times as long."""
    from nibble_b200 import _native

    count = _native.core().w4a16_launch_count
    torch.manual_seed(rows + n)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    spread = (torch.rand((n * (k // gs) + 1,), device="cuda") * 0.01 + 1e-3).half()
    row = torch.randn((rows * k + 1,), device="cuda").half()
    bias = torch.randn((n,), device="cuda").half()
    for shift_x, shift_scales in ((1, 0), (0, 1), (1, 1)):
        scales = spread[shift_scales:shift_scales + n * (k // gs)].view(n, k // gs)
        x = row[shift_x:shift_x + rows * k].view(1, rows, k)
        assert x.is_contiguous() and x.data_ptr() % 16 == 2 * shift_x and scales.data_ptr() % 16 == 2 * shift_scales
        product = torch.mm(x[0], torch.ops.w4a16.dequantize(packed, scales, gs).t())
        declined = shift_x or gs != 128
        for b in (None, bias):
            layer = QuantizedLinear(packed, scales, gs, bias=b)
            want = product if b is None else product + b
            before = count()
            got = layer(x)
            assert count() == before + 1 and got.shape == (1, rows, n)
            with _Passing():
                assert torch.equal(layer(x), got)
            if declined:
                assert torch.equal(got[0], want)
                with torch.autocast("cuda", dtype=torch.bfloat16):
                    assert torch.equal(torch.ops.w4a16.linear_bias(x, packed, scales, b, gs), got)
            else:
                torch.testing.assert_close(got[0], want, rtol=2e-3, atol=2e-3)
    torch._dynamo.reset()
    assert torch.equal(torch.compile(layer, backend="aot_eager", fullgraph=True, dynamic=False)(x), got)


@pytest.mark.parametrize(("variable", "value"), [("W4A16_DECODE", "generic"), ("W4A16_ROWS_PER_WARP", "2"), ("W4A16_ROWS_PER_WARP", "4")])
@pytest.mark.parametrize(("rows", "k", "n"), [(1025, 2048, 264), (2048, 8192, 1000), (1000, 1024, 4200), (300, 512, 10248)])
def test_variables_that_name_a_kernel_leave_large_batches_alone(variable, value, rows, k, n, monkeypatch):
    """They are for small and medium batches: beyond, the module's product is the one with dequantised weights, by its bits, where
    one of the kernels needs thirty times as long and the other refuses the call."""
    torch.manual_seed(rows)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    scales = (torch.rand((n, k // 128), device="cuda") * 0.01 + 1e-3).half()
    layer = QuantizedLinear(packed, scales, 128)
    x = torch.randn((rows, k), device="cuda").half()
    want = torch.mm(x, torch.ops.w4a16.dequantize(packed, scales, 128).t())
    monkeypatch.setenv(variable, value)
    assert torch.equal(layer(x), want)
    if value == "generic":                                   # on this side it is heeded: exact weights, another product's bits
        few = x[:100]
        product = torch.mm(few, torch.ops.w4a16.dequantize(packed, scales, 128).t())
        got = layer(few)
        assert not torch.equal(got, product)
        torch.testing.assert_close(got, product, rtol=1e-2, atol=1e-2 * float(product.abs().max()))


@pytest.mark.parametrize("rows", [4, 100])
def test_transforms_follow_the_product_with_dequantised_weights(rows):
    """Forward-mode differentiation and vmap see the matrix product where the module forms one."""
    from torch.autograd import forward_ad

    layer = _layer(n=64, k=256, seed=5)
    layer.fused = False
    w16 = torch.ops.w4a16.dequantize(layer.packed_weights, layer.scales, 128)
    x, direction = torch.randn((2, rows, 256), device="cuda").half()
    with forward_ad.dual_level():
        out = forward_ad.unpack_dual(layer(forward_ad.make_dual(x, direction)))
        assert out.tangent is not None
        torch.testing.assert_close(out.primal, F.linear(x, w16), rtol=1e-3, atol=1e-3)
        torch.testing.assert_close(out.tangent, F.linear(direction, w16), rtol=1e-3, atol=1e-3)
    batched = torch.vmap(layer)(torch.stack([x, direction]))
    torch.testing.assert_close(batched, torch.stack([layer(x), layer(direction)]), rtol=1e-3, atol=1e-3)
