"""The tile route with two row tiles per CTA (9 to 16 rows, one to two row tiles per SM): the bits of the streaming route's weights, an odd
number of row tiles, ragged N and K, gate/up pairs, and the give-up path."""
import ctypes

import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu
TILE = _native.ROUTE_TILE


def _layer(n, k, seed, kind="mixed"):
    g = torch.Generator(device="cuda").manual_seed(seed)
    sigma = 0.0006 if kind == "plain" else 0.02
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * sigma).half())
    if kind == "fp16":
        layer = ops.QuantizedLinear(layer.packed_weight, layer.scales.half().float(), layer.zeros, in_features=k)
    return layer, g


@pytest.mark.parametrize("m,n,k,kind", [(9, 2384, 2048, "mixed"), (16, 4736, 2048, "mixed"), (16, 2385, 1800, "plain"), (12, 3840, 4352, "mixed"),
                                        (10, 3828, 4104, "fp16"), (15, 3000, 3080, "plain"), (16, 4096, 4096, "fp16")])
def test_against_64_bit_sums(m, n, k, kind):
    layer, g = _layer(n, k, n + k, kind)
    image, flags = layer._native_image(), layer._image_flags
    assert _native.plan(m, 4096, 4096)["grid"] == 128
    x = torch.randn(m, k, generator=g, device="cuda").half()
    bias = torch.randn(n, generator=g, device="cuda").half()
    y = _native.linear(x, image, n, k, route=TILE, flags=flags)
    exact = x.double() @ layer.dequantize().half().double().t()
    assert ((y.double() - exact).abs() <= 2.0 ** -10 * exact.abs() + 1e-4).all()       # one rounding to FP16, FP32 sums
    assert torch.equal(_native.linear(x, image, n, k, route=TILE), y)
    assert torch.equal(_native.linear(x, image, n, k, route=TILE, bias=bias, flags=flags), y + bias)
    hot = torch.zeros(m, k, dtype=torch.float16, device="cuda")
    for i in range(m):
        hot[i, (i * 37 + k - 1) % k] = 1.0                                              # single weights, exactly
    columns = [(i * 37 + k - 1) % k for i in range(m)]
    assert torch.equal(_native.linear(hot, image, n, k, route=TILE, flags=flags), layer.dequantize().half()[:, columns].t())
    assert _native.status() == 0


def test_gate_up_pairs():
    m, n, k = 11, 4000, 2056
    layer, g = _layer(n, k, 3)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    lib, out = _native.load(), torch.zeros(m, n // 2, dtype=torch.float16, device="cuda")
    big = _native.linear(x, layer._native_image(), n, k)
    ws = torch.zeros(int(lib.b2_w4a16_workspace_bytes(m, n, k)), dtype=torch.uint8, device="cuda")
    assert lib.b2_w4a16_linear_silu_mul(x.data_ptr(), k, layer._native_image().data_ptr(), None, out.data_ptr(), n // 2, m, n, k, ws.data_ptr(),
                                        ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, _native.silu_mul_pairs(big))


def test_a_wait_that_runs_out():
    m, n, k = 16, 4096, 4096
    layer, g = _layer(n, k, 4)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    lib, image, word = _native.load(), layer._native_image(), ctypes.c_uint(7)
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")

    def call():
        y = torch.zeros(m, n, dtype=torch.float16, device="cuda")
        assert lib.b2_w4a16_linear_route(x.data_ptr(), k, image.data_ptr(), y.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(),
                                         torch.cuda.current_stream().cuda_stream, TILE) == 0
        assert lib.b2_w4a16_status(ws.data_ptr(), None, ctypes.byref(word)) == 0
        return y

    good = call()
    assert word.value == 0
    _native.test_hooks(wait_limit=64, skip_copy=3)
    try:
        call()
        assert word.value == 1
    finally:
        _native.test_hooks()
    ws.zero_()
    assert torch.equal(call(), good) and word.value == 0
