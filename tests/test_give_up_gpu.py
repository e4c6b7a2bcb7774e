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


@pytest.mark.parametrize("flags", [0, _native.FLAG_OVERLAP_LAUNCH])
@pytest.mark.parametrize("m,n,k,skipped,grid,parts", [
    (16, 5760, 16384, 0, 135, 3), (64, 12288, 8192, 9, 148, 3), (128, 24576, 4104, 3, 148, 2),                   # ranges
    (16, 24576, 2064, 1, 148, 3), (64, 20480, 3080, 0, 148, 7), (17, 20480, 3080, 9, 148, 7),                    # rounds, shared tiles first
    (20, 18952, 264, 0, 148, 1), (24, 16384, 520, 2, 128, 1), (60, 37888, 264, 3, 148, 1),                       # rounds of whole tiles
    (12, 16384, 4104, 4, 128, 1), (9, 1024, 4104, 1, 48, 6), (16, 8192, 1032, 2, 64, 1),                         # clusters, sixteen chains
    (17, 6144, 4096, 7, 96, 2), (100, 4096, 8200, 8, 128, 4), (129, 1000, 520, 1, 16, 1), (300, 1024, 2048, 0, 96, 4)])
def test_batch_kernel(m, n, k, skipped, grid, parts, flags):
    """The tickets of a shared tile are drawn, and the sums of a cluster waited for, after an abort too."""
    plan = _native.plan(m, n, k)
    assert plan["route"] == ("b200_batch" if m <= 128 else "b200_tcgen05") and plan["grid"] == grid and plan["k_splits"] == parts
    check(_native.ROUTE_AUTO, m, n, k, skipped, 2, flags=flags)
