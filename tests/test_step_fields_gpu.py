"""Step fields of the native image (csrc/layout.cuh): an FP32 step as the product of two FP16 numbers where that gives the same
sixteen weights, else as it is.  The fields must give the steps back bit for bit, and every kernel must use the very weights of
the format whichever form a group has."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu
SMALLEST, LARGEST = 2.0 ** -12, 3.99          # range of factored steps


def _state(n, k, seed):
    """Random steps over the whole FP32 range and around the ends of the factored range; every zero point."""
    g = torch.Generator().manual_seed(seed)
    groups = -(-k // 64)
    codes = torch.randint(0, 16, (n, k), generator=g, dtype=torch.uint8)
    zeros = torch.randint(0, 16, (n, groups), generator=g, dtype=torch.int32)
    steps = torch.exp(torch.randn(n, groups, generator=g) - 5.0)
    kind = torch.randint(0, 8, (n, groups), generator=g)
    steps = torch.where(kind == 1, steps.half().float(), steps)
    steps = torch.where(kind == 2, torch.exp(torch.rand(n, groups, generator=g) * 160 - 85), steps)
    edge = torch.tensor([SMALLEST, LARGEST]).view(torch.int32)[torch.randint(0, 2, (n, groups), generator=g)]
    edge = (edge + torch.randint(-2, 3, (n, groups), generator=g, dtype=torch.int32)).view(torch.float32)
    steps = torch.where(kind == 3, edge, steps)
    return ops.pack_int4(codes.cuda()), steps.cuda(), zeros.cuda()


def _fields(image):
    return image.view(-1, 2336)[:, 2048:2304].contiguous().view(torch.int32)


@pytest.mark.parametrize("n,k", [(16, 256), (100, 520), (1000, 4096)])
def test_round_trip_and_share_of_factored_groups(n, k):
    packed, steps, zeros = _state(n, k, n + k)
    image = _native.repack(packed, steps, zeros, k)
    for got, want in zip(_native.unrepack(image, n, k), (packed, steps, zeros)):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert torch.equal(_native.dequantize(image, n, k).view(torch.int32), ops.dequantize_int4(packed, steps, zeros, k).view(torch.int32))
    weight = (torch.randn(n, k, generator=torch.Generator().manual_seed(k)) * 0.02).half().cuda()
    assert (_fields(ops.QuantizedLinear.from_float(weight)._native_image()) < 0).float().mean() > 0.995


def test_a_negative_step_gives_the_same_weights():
    packed, steps, zeros = _state(64, 256, 9)
    steps[::3] *= -1
    image = _native.repack(packed, steps, zeros, 256)
    assert torch.equal(_native.dequantize(image, 64, 256), ops.dequantize_int4(packed, steps, zeros, 256))


# tile, streaming with one to eight row tiles of x and with unaligned x, batch kernel, single-CTA and pair GEMM, whatever
# the automatic choice is at 520 rows
@pytest.mark.parametrize("shape,route,m,n,k", [
    ("auto", _native.ROUTE_TILE, 8, 1000, 520), ("auto", _native.ROUTE_TILE, 16, 48, 2048),
    ("auto", _native.ROUTE_STREAM, 1, 1000, 1000), ("auto", _native.ROUTE_STREAM, 16, 1000, 520), ("auto", _native.ROUTE_STREAM, 64, 600, 257),
    ("auto", _native.ROUTE_BATCH, 16, 1000, 520), ("auto", _native.ROUTE_BATCH, 128, 600, 1032),
    ("128x128", _native.ROUTE_TCGEN05, 128, 300, 520), ("pair256", _native.ROUTE_TCGEN05, 256, 300, 520), ("pair192", _native.ROUTE_TCGEN05, 192, 300, 520),
    ("auto", _native.ROUTE_TCGEN05, 520, 700, 520)])
def test_weights_in_the_kernels_are_exact(shape, route, m, n, k):
    """One-hot rows of x read single weight columns: y[m, n] must be fp16(w[n, column m])."""
    packed, steps, zeros = _state(n, k, n + k + m)
    steps.clamp_(max=4.0e3)                                   # (finite FP16 weights)
    image = _native.repack(packed, steps, zeros, k)
    weights = ops.dequantize_int4(packed, steps, zeros, k).half()
    _native.set_gemm_shape(shape)
    try:
        for first in range(0, k, m):
            columns = torch.arange(first, min(first + m, k), device="cuda")
            x = torch.zeros(m, k, dtype=torch.float16, device="cuda")
            x[torch.arange(len(columns), device="cuda"), columns] = 1.0
            y = _native.linear(x, image, n, k, route=route)
            assert torch.equal(y[: len(columns)], weights[:, columns].t())
    finally:
        _native.set_gemm_shape("auto")
    assert _native.status() == 0
