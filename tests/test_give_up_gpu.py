"""Waits that run out, in every form of the decode kernels: one weight copy of the first CTA is left out (its barrier is armed), the
warps that need it give up, the call returns with the status word set, and the next call is right."""
import ctypes

import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu
TILE, STREAM = _native.ROUTE_TILE, _native.ROUTE_STREAM


def check(route, m, n, k, skipped, bit, offset=0, flags=0):
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * 0.02).half())
    x = torch.randn(m * k + offset, generator=g, device="cuda").half()[offset:].view(m, k)
    lib, image, word = _native.load(), layer._native_image(), ctypes.c_uint(7)
    ws = torch.zeros(int(lib.b2_w4a16_workspace_bytes(m, n, k)), dtype=torch.uint8, device="cuda")

    def call():
        y = torch.zeros(m, n, dtype=torch.float16, device="cuda")
        assert lib.b2_w4a16_linear_flags(x.data_ptr(), k, image.data_ptr(), None, y.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(),
                                         torch.cuda.current_stream().cuda_stream, route, flags) == 0, lib.b2_w4a16_last_error()
        assert lib.b2_w4a16_status(ws.data_ptr(), None, ctypes.byref(word)) == 0
        return y

    good = call()
    assert word.value == 0
    _native.test_hooks(wait_limit=64, skip_copy=skipped)
    try:
        call()
        assert word.value == bit
    finally:
        _native.test_hooks()
    ws.zero_()
    assert torch.equal(call(), good) and word.value == 0


@pytest.mark.parametrize("flags", [0, _native.FLAG_OVERLAP_LAUNCH])
@pytest.mark.parametrize("m,n,k,offset,skipped", [(1, 4096, 1024, 0, 3), (8, 6144, 1032, 0, 0), (16, 2048, 1024, 0, 2), (3, 3000, 2056, 1, 8),
                                                  (4, 1024, 2048, 0, 3), (16, 512, 8192, 0, 7), (16, 4096, 4096, 0, 15)])
def test_tile_kernel(m, n, k, offset, skipped, flags):
    check(TILE, m, n, k, skipped, 1, offset, flags)


@pytest.mark.parametrize("flags", [0, _native.FLAG_OVERLAP_LAUNCH])
@pytest.mark.parametrize("m,n,k,offset,skipped", [(1, 512, 1024, 0, 0), (4, 8192, 4096, 0, 1), (8, 12288, 2048, 0, 1), (16, 12288, 2056, 0, 0),
                                                  (24, 8192, 4096, 1, 1), (64, 2048, 4096, 1, 0)])
def test_streaming_kernel(m, n, k, offset, skipped, flags):
    check(STREAM, m, n, k, skipped, 1, offset, flags)
