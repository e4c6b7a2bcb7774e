"""Layers that the tile route splits along K: the sums of a cluster's CTAs meet in the first one's shared memory, counted on a barrier
that has to be set up before any of them is sent."""
import ctypes

import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu
TILE = _native.ROUTE_TILE


def _layer(n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    return ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * 0.02).half()), g


@pytest.mark.parametrize("m,n,k,parts", [(1, 1024, 2048, 2), (8, 1001, 2056, 2), (9, 1184, 2048, 2), (16, 1024, 3080, 2), (5, 592, 4096, 4),
                                         (16, 512, 8192, 4), (3, 16, 4104, 4)])
def test_hand_over(m, n, k, parts):
    """Peers whose weights come from L2 are through soonest: many launches in a row, each as early as it may start."""
    layer, g = _layer(n, k)
    image, flags = layer._native_image(), layer._image_flags | _native.FLAG_OVERLAP_LAUNCH
    if (plan := _native.plan(m, n, k))["route"] == "b200_tile":
        assert plan["k_splits"] == parts and plan["grid"] == -(-n // 16) * parts
    x = torch.randn(m, k, generator=g, device="cuda").half()
    y = _native.linear(x, image, n, k, route=TILE)
    exact = x.double() @ layer.dequantize().half().double().t()
    assert ((y.double() - exact).abs() <= 2.0 ** -10 * exact.abs() + 1e-4).all()       # one rounding to FP16, FP32 sums
    outs = [torch.full_like(y, 7.0) for _ in range(64)]
    for _ in range(8):
        for out in outs:
            _native.linear(x, image, n, k, route=TILE, flags=flags, out=out)
        assert all(torch.equal(out, y) for out in outs)
    assert _native.status() == 0


@pytest.mark.parametrize("m,n,k,skipped", [(1, 1024, 2048, 0), (16, 1024, 3080, 5), (8, 512, 8192, 7)])
def test_a_wait_that_runs_out(m, n, k, skipped):
    layer, g = _layer(n, k)
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
    _native.test_hooks(wait_limit=64, skip_copy=skipped)
    try:
        call()
        assert word.value == 1
    finally:
        _native.test_hooks()
    ws.zero_()
    assert torch.equal(call(), good) and word.value == 0
