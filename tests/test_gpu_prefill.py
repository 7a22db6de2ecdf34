"""-m gpu: prefill-sized batches (M >= 65) take one of the two tcgen05 GEMMs that dequantise into tensor memory.  Checked against the oracle on the same packed codes, against the mma.sync kernel,
and for a clean device status word (no barrier wait gave up)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from capi_helpers import capi_dequantize, capi_linear, check_against_oracle, kernels_of, new_workspace
from nibble_b200 import _native, quantize_and_pack_weights
from oracle import w4a16_oracle as oracle

pytestmark = pytest.mark.gpu


def _device_status() -> int:
    value = ctypes.c_uint32(123)
    assert _native.core().w4a16_device_status(ctypes.byref(value)) == 0
    return value.value


def _gemm_of(call) -> str:
    """Which GEMM one call takes: "single" SMs or "pair"."""
    names = [name for name in kernels_of(call) if "linear_" in name]
    assert len(names) == 1, names
    assert "linear_gemm_kernel" in names[0] or "linear_gemm_pair_kernel" in names[0], names
    return "pair" if "linear_gemm_pair_kernel" in names[0] else "single"


def _case(m, k, n, seed):
    g = torch.Generator().manual_seed(seed)
    w = torch.randn((n, k), generator=g) * 0.02
    x = torch.randn((m, k), generator=g).half()
    packed, scales = quantize_and_pack_weights(w, 128)
    return x.cuda(), packed.cuda(), scales.cuda()


@pytest.mark.parametrize("m", [65, 128, 129, 300])
@pytest.mark.parametrize(("k", "n"), [(128, 128), (512, 256), (1024, 250), (2048, 2048), (5632, 384)])
def test_tcgen05_path_matches_oracle(m, k, n):
    _device_status()   # clear
    x, packed, scales = _case(m, k, n, seed=m + k + n)
    before = _native.core().w4a16_launch_count()
    y = capi_linear(x, packed, scales)
    torch.cuda.synchronize()
    assert _device_status() == 0, "a barrier wait inside the tcgen05 kernel gave up"
    assert _native.core().w4a16_launch_count() == before + 1
    check_against_oracle(y, x, packed, scales)
    # the product of FP16-rounded weights, FP32 accumulate: what dequantise-then-matmul computes
    w16 = oracle.dequantize_weights(packed.cpu().numpy(), scales.cpu().numpy(), 128).astype(np.float16)
    ref = torch.from_numpy(x.cpu().numpy().astype(np.float32) @ w16.astype(np.float32).T)
    torch.testing.assert_close(y.float().cpu(), ref, rtol=2e-3, atol=2e-3)
    # and the streaming mma.sync kernel on the same inputs
    other = capi_linear(x, packed, scales, flags=_native.FLAG_NO_TCGEN05)
    torch.testing.assert_close(y, other, rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize(("m", "k", "n"), [
    (600, 512, 8192),      # pairs of SMs, 3 x 32 tiles: two for some
    (1024, 256, 16384),    # 256 tiles: at least three a pair
    (257, 1024, 1000),     # two ragged batch tiles, ragged last weight slab
    (2048, 2048, 640),     # single SMs, 16 batch tiles
])
def test_tcgen05_many_tiles(m, k, n):
    _device_status()
    x, packed, scales = _case(m, k, n, seed=m ^ n)
    y = capi_linear(x, packed, scales)
    torch.cuda.synchronize()
    assert _device_status() == 0
    w16 = torch.from_numpy(oracle.dequantize_weights(packed.cpu().numpy(), scales.cpu().numpy(), 128).astype(np.float16))
    ref = (x.float() @ w16.cuda().float().t())
    torch.testing.assert_close(y.float(), ref, rtol=2e-3, atol=2e-3)
    rows = np.random.default_rng(m).choice(n, size=64, replace=False)
    check_against_oracle(y, x, packed, scales, rows=np.sort(rows), fp16_weights=True)


@pytest.mark.parametrize(("m", "k", "n"), [
    (17, 384, 128),       # single SMs: three blocks, one for each group of dequantisers
    (40, 640, 256),       # five
    (64, 1152, 384),      # nine, two tiles
    (128, 896, 200),      # pairs of SMs: seven, for four groups
    (130, 640, 128),      # five; one SM of the pair has no channel
    (256, 384, 256),      # single SMs, two batch tiles
    (200, 128, 128),      # one block
])
def test_forced_gemm_on_odd_block_counts(m, k, n):
    """K blocks that do not come out even among the groups of dequantisers, through the flag that sends any batch to a GEMM."""
    _device_status()
    x, packed, scales = _case(m, k, n, seed=m * 7 + k)
    y = capi_linear(x, packed, scales, flags=_native.FLAG_FORCE_TCGEN05)
    torch.cuda.synchronize()
    assert _device_status() == 0
    check_against_oracle(y, x, packed, scales, fp16_weights=True)
    again = capi_linear(x, packed, scales, flags=_native.FLAG_FORCE_TCGEN05)
    assert torch.equal(y, again)


@pytest.mark.parametrize("m", [16, 17, 33, 64])
def test_medium_batches_on_a_large_layer_take_the_gemm(m):
    """A layer of K = 8192, N = 4096 is cheaper on the GEMM than on the streaming kernel from 17 rows on: the default
    route then gives what the forced GEMM gives, bit for bit; up to 16 rows, what the streaming kernel gives.  The
    two agree within the tolerance."""
    k, n = 8192, 4096
    takes_gemm = m > 16        # the cost model's verdict for this layer; the bit comparison below pins it
    _device_status()
    x, packed, scales = _case(m, k, n, seed=m)
    ws = new_workspace(m, n, k)
    y = capi_linear(x, packed, scales, workspace=ws)
    forced = capi_linear(x, packed, scales, workspace=ws, flags=_native.FLAG_FORCE_TCGEN05)
    streaming = capi_linear(x, packed, scales, workspace=ws, flags=_native.FLAG_NO_TCGEN05)
    torch.cuda.synchronize()
    assert _device_status() == 0
    assert torch.equal(y, forced if takes_gemm else streaming)
    torch.testing.assert_close(forced, streaming, rtol=1e-2, atol=1e-2)
    rows = np.sort(np.random.default_rng(m).choice(n, size=32, replace=False))
    check_against_oracle(forced, x, packed, scales, rows=rows, fp16_weights=True)


def test_batch_too_large_for_the_streaming_kernel_without_scratch_takes_the_gemm():
    """32 rows of K = 28672 do not fit one CTA's shared memory unsplit; without a workspace the call used to fall
    to the generic kernel (milliseconds) and now runs the GEMM."""
    m, k, n = 32, 28672, 256
    _device_status()
    x, packed, scales = _case(m, k, n, seed=5)
    y = capi_linear(x, packed, scales, workspace=None)
    forced = capi_linear(x, packed, scales, flags=_native.FLAG_FORCE_TCGEN05)
    torch.cuda.synchronize()
    assert _device_status() == 0
    assert torch.equal(y, forced)
    check_against_oracle(y, x, packed, scales, fp16_weights=True)


@pytest.mark.parametrize(("m", "k", "n"), [
    (65, 4096, 256),       # 1 tile: eight CTAs share its 32 blocks
    (65, 4096, 250),       # the same, ragged channels
    (128, 4096, 1024),     # 4 tiles
    (100, 4352, 640),      # 3 tiles of 34 blocks: shares of four and five
    (300, 8192, 512),      # three batch tiles, 6 tiles in all
    (32, 8192, 4096),      # a medium batch on the forced GEMM: 16 tiles
])
def test_gemm_splits_k_when_the_layer_has_few_tiles(m, k, n):
    """Layers of few tiles, whose K the GEMM shares between CTAs (inside clusters, so that a workspace changes nothing):
    with the workspace the query names, with none and with one too small.  All agree with the oracle, and the workspace's
    counter prefix, which the streaming kernel relies on, is left at zero."""
    lib = _native.core()
    flags = _native.FLAG_FORCE_TCGEN05
    need = lib.w4a16_linear_workspace_bytes_flags(m, n, k, flags)
    assert need > 256 * 1024, "this layer should want K split"
    _device_status()
    x, packed, scales = _case(m, k, n, seed=m + n)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    split = capi_linear(x, packed, scales, workspace=ws, flags=flags)
    again = capi_linear(x, packed, scales, workspace=ws, flags=flags)
    unsplit = capi_linear(x, packed, scales, flags=flags)
    torch.cuda.synchronize()
    assert _device_status() == 0
    assert torch.equal(split, again)
    torch.testing.assert_close(split, unsplit, rtol=2e-3, atol=2e-3)
    check_against_oracle(split, x, packed, scales, fp16_weights=True)
    assert int(ws[: 256 * 1024].sum()) == 0
    # a workspace that is too small is not an error: the GEMM runs unsplit
    small = torch.zeros(256 * 1024 + 64, dtype=torch.uint8, device="cuda")
    assert torch.equal(capi_linear(x, packed, scales, workspace=small, flags=flags), unsplit)


def test_all_nibble_values_and_repeatability(golden):
    data = golden("all_nibbles.npz")
    packed = torch.from_numpy(data["packed"]).cuda()
    scales = torch.from_numpy(data["scales"]).cuda()
    x = torch.randn((96, 1024), generator=torch.Generator().manual_seed(5)).half().cuda()
    for rows, gemm in ((96, "pair"), (64, "single")):
        some = x[:rows]
        first = capi_linear(some, packed, scales, flags=_native.FLAG_FORCE_TCGEN05)
        assert _gemm_of(lambda: capi_linear(some, packed, scales, flags=_native.FLAG_FORCE_TCGEN05)) == gemm
        assert torch.equal(capi_linear(some, packed, scales, flags=_native.FLAG_FORCE_TCGEN05), first)
        assert _device_status() == 0
        check_against_oracle(first, some, packed, scales, fp16_weights=True)


@pytest.mark.parametrize(("m", "k", "n", "gs"), [
    (40, 1024, 1000, 128),     # few tiles: a cluster per tile
    (65, 4096, 1900, 128),     # batch tile above 64 rows: two weight slots
    (128, 8192, 28672, 128),   # equal runs that cut tiles, two segments each
    (40, 8192, 28672, 128),    # ... with three weight slots
    (100, 5632, 19001, 128),   # ... on ragged channels
    (300, 512, 20000, 128),    # runs of several whole tiles, three batch tiles
    (777, 1024, 5376, 128),    # 147 whole tiles
    (128, 4096, 3000, 64), (300, 8192, 1000, 32), (77, 2048, 32000, 32),
])
def test_gemm_on_single_sms(m, k, n, gs):
    """Every way this GEMM shares tiles, with and without a workspace, against the product with the same FP16 weights."""
    from nibble_b200 import dequantize_cuda

    _device_status()
    g = torch.Generator(device="cuda").manual_seed(m + k)
    packed, scales = quantize_and_pack_weights(torch.randn((n, k), generator=g, device="cuda") * 0.02, gs)
    x = torch.randn((m, k), generator=g, device="cuda").half()
    want = x.float() @ dequantize_cuda(packed, scales, gs).float().t()
    ws = torch.zeros(40 << 20, dtype=torch.uint8, device="cuda")
    for workspace in (ws, ws, None):
        assert _gemm_of(lambda: capi_linear(x, packed, scales, gs, workspace=workspace, flags=_native.FLAG_FORCE_TCGEN05)) == "single"
        y = capi_linear(x, packed, scales, gs, workspace=workspace, flags=_native.FLAG_FORCE_TCGEN05)
        torch.testing.assert_close(y.float(), want, rtol=2e-3, atol=2e-3)
        assert torch.equal(y, capi_linear(x, packed, scales, gs, workspace=workspace, flags=_native.FLAG_FORCE_TCGEN05))
    assert int(ws[: 256 * 1024].sum()) == 0
    assert _device_status() == 0, "a barrier wait gave up"


@pytest.mark.parametrize(("m", "k", "n", "gs"), [(128, 8192, 28672, 128), (40, 8192, 28672, 128), (120, 8192, 25001, 32),
                                                 (128, 8192, 28672, 64)])
def test_scratch_query_is_exact_for_equal_runs(m, k, n, gs):
    """With the bytes the query names the GEMM does what it does with any more; with one less, what it does without."""
    lib = _native.core()
    flags = _native.FLAG_FP16_WEIGHTS
    need = lib.w4a16_linear_scratch_bytes(m, n, k, gs, flags)
    assert need > 256 * 1024
    torch.manual_seed(m + n)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    scales = (torch.rand((n, k // gs), device="cuda") * 0.01 + 1e-3).half()
    x = torch.randn((m, k), device="cuda").half()

    def run(size):
        workspace = None if size is None else torch.zeros(size, dtype=torch.uint8, device="cuda")
        return capi_linear(x, packed, scales, gs, workspace=workspace, flags=flags)

    shared, whole = run(need), run(None)
    assert torch.equal(run(40 << 20), shared) and torch.equal(run(need - 1), whole)
    torch.testing.assert_close(shared, whole, rtol=2e-3, atol=2e-3)
    assert _device_status() == 0


@pytest.mark.parametrize("gs", [128, 64, 32])
@pytest.mark.parametrize(("m", "k", "n", "gemm"), [
    (128, 8192, 28672, "single"), (64, 8192, 16384, "single"), (100, 28672, 8192, "single"), (300, 5632, 12345, "single"),
    (2048, 8192, 28672, "pair"), (512, 2048, 5000, "pair"), (700, 640, 12000, "pair"),
])
def test_gemm_results_do_not_depend_on_timing(m, k, n, gemm, gs):
    """Forty calls, with other work in front of some of them, give the bits of the first: a slot of codes refilled while a
    dequantiser still reads it shows as a few wrong output channels in one call out of many."""
    torch.manual_seed(m + gs)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    scales = (torch.rand((n, k // gs), device="cuda") * 0.01 + 1e-3).half()
    x = torch.randn((m, k), device="cuda").half()
    flags = _native.FLAG_FORCE_TCGEN05
    for workspace in (None, torch.zeros(40 << 20, dtype=torch.uint8, device="cuda")):
        first = capi_linear(x, packed, scales, gs, workspace=workspace, flags=flags)
        assert _gemm_of(lambda: capi_linear(x, packed, scales, gs, workspace=workspace, flags=flags)) == gemm
        different = 0
        for call in range(40):
            if call % 4 == 3:
                _ = x.float() @ x.float().t()
            different += int((capi_linear(x, packed, scales, gs, workspace=workspace, flags=flags) != first).any())
        assert different == 0
    from nibble_b200 import dequantize_cuda
    torch.testing.assert_close(first.float(), x.float() @ dequantize_cuda(packed, scales, gs).float().t(), rtol=2e-3, atol=1e-2)
    assert _device_status() == 0


@pytest.mark.parametrize(("m", "k", "n", "gemm"), [
    (64, 2048, 18944, None), (128, 2048, 18944, "pair"), (128, 2048, 18945, "single"),          # 74 and 75 tiles of pairs
    (777, 1024, 5376, "single"), (777, 1024, 5377, "pair"),                                     # 147 and 154 of single SMs
    (1024, 2048, 9728, "single"), (1025, 2048, 9728, "pair"), (1024, 1920, 9728, "pair"),
    (2500, 3968, 1930, "pair"), (2500, 4096, 1930, "single"),                                   # 160
    (2048, 4096, 4700, "pair"),                                                                 # 304
    (2048, 4096, 4000, "pair"), (5000, 4096, 1000, "single"), (3000, 256, 130, "single"),       # by their models
])
def test_either_side_of_the_lines_between_the_gemms(m, k, n, gemm):
    """The kernel that each side of each line names runs there, and gives the product with the same FP16 weights, the same bits again,
    and nothing outside the output."""
    from nibble_b200 import dequantize_cuda

    _device_status()
    torch.manual_seed(m + n)
    packed, scales = quantize_and_pack_weights(torch.randn((n, k), device="cuda") * 0.02, 128)
    x = torch.randn((m, k), device="cuda").half()
    want = x.float() @ dequantize_cuda(packed, scales, 128).float().t()
    need = _native.core().w4a16_linear_scratch_bytes(m, n, k, 128, 0)
    for workspace in (None, torch.zeros(max(need, 16), dtype=torch.uint8, device="cuda")):
        y = capi_linear(x, packed, scales, workspace=workspace)
        if gemm is not None and (workspace is not None or need == 0):      # (64 rows stream or not by a line of their own)
            assert _gemm_of(lambda: capi_linear(x, packed, scales, workspace=workspace)) == gemm
        torch.testing.assert_close(y.float(), want, rtol=2e-3, atol=2e-3)
        assert torch.equal(y, capi_linear(x, packed, scales, workspace=workspace))
    assert _device_status() == 0


@pytest.mark.parametrize(("m", "k", "n"), [
    (65, 128, 9600), (128, 384, 9601), (96, 640, 18944), (100, 896, 12345), (128, 1024, 9473), (66, 1024, 18943),
    (513, 384, 16385), (700, 640, 12000), (1100, 896, 9001), (1025, 1152, 9216), (2049, 2048, 2500), (2500, 3968, 1930), (2000, 5632, 4900),
])
def test_gemms_on_ragged_layers(m, k, n):
    """Odd numbers of K blocks, ragged channels and batches, with and without a bias; one launch, no scratch."""
    from nibble_b200 import dequantize_cuda

    lib = _native.core()
    assert lib.w4a16_linear_scratch_bytes(m, n, k, 128, 0) == 0
    _device_status()
    torch.manual_seed(m + k)
    packed, scales = quantize_and_pack_weights(torch.randn((n, k), device="cuda") * 0.02, 128)
    x = torch.randn((m, k), device="cuda").half()
    want = x.float() @ dequantize_cuda(packed, scales, 128).float().t()
    before = lib.w4a16_launch_count()
    y = capi_linear(x, packed, scales)
    assert lib.w4a16_launch_count() == before + 1
    torch.testing.assert_close(y.float(), want, rtol=2e-3, atol=2e-3)
    for _ in range(10):
        assert torch.equal(capi_linear(x, packed, scales), y)
    bias = torch.randn((n,), device="cuda").half()
    assert torch.equal(torch.ops.w4a16.linear_bias(x, packed, scales, bias, 128), y + bias)
    assert _device_status() == 0


@pytest.mark.parametrize("gs", [128, 64, 32])
def test_gemm_weights_are_rounded_products_for_any_scale(gs):
    """Single ones as activations read the weights of both GEMMs out: half(code * scale) whatever the scale, either side of the line
    where warps of small scales take an FMA on (code + 8) * 2^-20 (its largest scale is 65504 / 2^20, FP16 bits 0x2BFF)."""
    k, n = 512, 300
    g = torch.Generator().manual_seed(gs)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, generator=g).cuda()
    bits = torch.randint(1, 0x2BFF, (n, k // gs), generator=g)                       # subnormal scales among them
    edges = torch.tensor([0x0001, 0x03FF, 0x0400, 0x2BFE, 0x2BFF, 0x2C00, 0x3C00, 0x6B00, 0x0000, 0xABFF, 0xAC00, 0x8001])
    bits[64:128] = edges[torch.randint(0, len(edges), (64, k // gs), generator=g)]   # mixed in two warps of a tile
    bits[128:192] = torch.where(bits[128:192] % 2 == 0, 0x2BFF, 0xABFF)              # on the line, in all of them
    scales = bits.to(torch.int16).view(torch.float16).cuda()
    weights = capi_dequantize(packed, scales, gs)
    flags = _native.FLAG_FORCE_TCGEN05
    _device_status()
    for rows, gemm in ((128, "pair"), (64, "single")):
        for first in range(0, k, rows):
            x = torch.zeros((rows, k), dtype=torch.float16, device="cuda")
            x[torch.arange(rows), first + torch.arange(rows)] = 1.0
            y = capi_linear(x, packed, scales, gs, flags=flags)
            torch.testing.assert_close(y, weights[:, first:first + rows].t(), rtol=0, atol=0)
        assert _gemm_of(lambda: capi_linear(x, packed, scales, gs, flags=flags)) == gemm
    assert _device_status() == 0


@pytest.mark.parametrize(("m", "k", "n", "gs"), [
    (65, 1024, 513, 128),      # 96 rows, 48 to an SM; one channel in the last tile, none for its second SM
    (128, 384, 300, 128),      # fewer blocks than weight slots
    (96, 2048, 12000, 128), (200, 2048, 18900, 128),   # one tile a pair; codes and x go round their rings
    (700, 640, 12000, 128),    # three batch tiles of 256; two tiles and more a pair: the accumulator is handed back
    (1500, 2048, 4096, 128), (1100, 384, 9001, 128),
    (3000, 128, 5000, 128),    # one K block a tile
    (2050, 256, 2500, 128),
    (2600, 256, 2300, 128), (4900, 128, 1030, 128),    # bands of 6 and 5, of 7, 7 and 6 batch tiles
    (1030, 896, 2000, 64), (1300, 640, 5001, 64), (2100, 384, 3100, 32),
])
def test_gemm_on_pairs_of_sms(m, k, n, gs):
    """Calls that the pair kernel takes (they need no scratch), against the product with the same FP16 weights, with and without a
    bias; the same bits again, and nothing outside the output."""
    from nibble_b200 import dequantize_cuda

    lib, flags = _native.core(), _native.FLAG_FP16_WEIGHTS
    assert lib.w4a16_linear_scratch_bytes(m, n, k, gs, flags) == 0
    _device_status()
    torch.manual_seed(m + k)
    packed, scales = quantize_and_pack_weights(torch.randn((n, k), device="cuda") * 0.02, gs)
    x = torch.randn((m, k), device="cuda").half()
    want = x.float() @ dequantize_cuda(packed, scales, gs).float().t()
    before = lib.w4a16_launch_count()
    y = capi_linear(x, packed, scales, gs, flags=flags)
    assert lib.w4a16_launch_count() == before + 1
    assert _gemm_of(lambda: capi_linear(x, packed, scales, gs, flags=flags)) == "pair"
    # FP32 sums in two orders, each within K * 2^-24 of the products' magnitudes, and one rounding to FP16
    torch.testing.assert_close(y.float(), want, rtol=2e-3, atol=2e-3)
    for _ in range(10):
        assert torch.equal(capi_linear(x, packed, scales, gs, flags=flags), y)
    bias = torch.randn((n,), device="cuda").half()
    assert torch.equal(torch.ops.w4a16.linear_bias(x, packed, scales, bias, gs), y + bias)
    assert _device_status() == 0


@pytest.mark.parametrize(("m", "k", "n"), [(300, 8192, 28672), (384, 4096, 14336)])
def test_the_gemm_is_chosen_by_what_the_workspace_allows(m, k, n):
    """Equal runs that cut tiles are what makes single SMs the faster way for these layers: a call without room for the parts
    takes pairs, whatever the room would have allowed."""
    lib = _native.core()
    need = lib.w4a16_linear_scratch_bytes(m, n, k, 128, 0)
    assert need > 4 << 20
    torch.manual_seed(m)
    packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda")
    scales = (torch.rand((n, k // 128), device="cuda") * 0.01 + 1e-3).half()
    x = torch.randn((m, k), device="cuda").half()
    workspace = torch.zeros(need + 16, dtype=torch.uint8, device="cuda")
    results = {}
    for name, given in (("enough", workspace[:need]), ("too small", workspace[:need - 1]), ("misaligned", workspace[8:need + 8]), ("none", None)):
        results[name] = capi_linear(x, packed, scales, workspace=given)
        assert _gemm_of(lambda: capi_linear(x, packed, scales, workspace=given)) == ("single" if name == "enough" else "pair"), name
    assert torch.equal(results["too small"], results["none"]) and torch.equal(results["misaligned"], results["none"])
    torch.testing.assert_close(results["enough"], results["none"], rtol=2e-3, atol=1e-2)
    assert _device_status() == 0
