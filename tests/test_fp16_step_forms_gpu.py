"""Layers whose steps FP16 can hold, with steps on both sides of the factored range (csrc/layout.cuh): FP16 subnormals and steps
of 4 and more keep plain fields, the others are factored, and most blocks hold both forms.  Every kernel must read
the very weights of the format from them, with B2_FLAG_FP16_STEPS (one chain for both forms) and without it."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu


def _state(n, k, seed):
    g = torch.Generator().manual_seed(seed)
    groups = -(-k // 64)
    codes = torch.randint(0, 16, (n, k), generator=g, dtype=torch.uint8)
    zeros = torch.randint(0, 16, (n, groups), generator=g, dtype=torch.int32)
    steps = torch.exp(torch.randn(n, groups, generator=g) * 0.5 - 5.0)
    kind = torch.randint(0, 14, (n, groups), generator=g)
    steps = torch.where(kind == 1, torch.exp2(-24 + 14 * torch.rand(n, groups, generator=g)), steps)      # from FP16's smallest number on
    steps = torch.where(kind == 2, 4.0 + 4000.0 * torch.rand(n, groups, generator=g), steps)
    steps = steps.half().float().clamp_min(2.0 ** -24)
    return ops.pack_int4(codes.cuda()), steps.cuda(), zeros.cuda()


@pytest.mark.parametrize("shape,route,m,n,k", [
    ("auto", _native.ROUTE_TILE, 1, 1000, 520), ("auto", _native.ROUTE_TILE, 8, 1000, 520), ("auto", _native.ROUTE_TILE, 16, 48, 2048),
    ("auto", _native.ROUTE_STREAM, 1, 1000, 1000), ("auto", _native.ROUTE_STREAM, 8, 600, 1024), ("auto", _native.ROUTE_STREAM, 16, 1000, 520),
    ("auto", _native.ROUTE_STREAM, 64, 600, 520), ("auto", _native.ROUTE_BATCH, 16, 1000, 520), ("auto", _native.ROUTE_BATCH, 128, 600, 1032),
    ("pair256", _native.ROUTE_TCGEN05, 256, 304, 520), ("pair192", _native.ROUTE_TCGEN05, 192, 304, 520),
    ("128x128", _native.ROUTE_TCGEN05, 128, 300, 520)])
def test_both_forms_of_fp16_steps_give_the_weights(shape, route, m, n, k):
    """One-hot rows of x read single weight columns: y[m, n] must be fp16(w[n, column m])."""
    packed, steps, zeros = _state(n, k, n + k + m)
    image = _native.repack(packed, steps, zeros, k)
    factored = image.view(-1, 2336)[:, 2048:2304].contiguous().view(torch.int32) < 0
    assert (factored.any(1) & ~factored.all(1)).float().mean() > 0.4                    # blocks with both forms
    weights = ops.dequantize_int4(packed, steps, zeros, k).half()
    assert torch.isfinite(weights).all()
    _native.set_gemm_shape(shape)
    try:
        for flags in (0, _native.FLAG_FP16_STEPS):
            for first in range(0, k, m):
                columns = torch.arange(first, min(first + m, k), device="cuda")
                x = torch.zeros(m, k, dtype=torch.float16, device="cuda")
                x[torch.arange(len(columns), device="cuda"), columns] = 1.0
                y = _native.linear(x, image, n, k, route=route, flags=flags)
                assert torch.equal(y[: len(columns)], weights[:, columns].t())
    finally:
        _native.set_gemm_shape("auto")
    assert _native.status() == 0
