"""Steps that are negative (no checkpoint holds one, but the C entry points take them): the image keeps a group as the equal one
with the step's absolute value and codes and zero point subtracted from 15."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu


def _state(n, k):
    g = torch.Generator().manual_seed(n + k)
    groups = -(-k // 64)
    codes = torch.randint(0, 16, (n, k), generator=g, dtype=torch.uint8)
    zeros = torch.randint(0, 16, (n, groups), generator=g, dtype=torch.int32)
    steps = torch.exp(torch.randn(n, groups, generator=g) - 5.0)
    steps = torch.where(torch.rand(n, groups, generator=g) < 0.2, steps * 1e-3, steps)            # some below the factored range
    steps = torch.where(torch.rand(n, groups, generator=g) < 0.4, -steps, steps)
    return codes, steps, zeros


@pytest.mark.parametrize("n,k", [(64, 256), (100, 520)])
def test_unrepack_returns_the_equal_state(n, k):
    codes, steps, zeros = _state(n, k)
    image = _native.repack(ops.pack_int4(codes.cuda()), steps.cuda(), zeros.cuda(), k)
    packed, got_steps, got_zeros = _native.unrepack(image, n, k)
    negative = steps < 0
    by_column = negative.repeat_interleave(64, dim=1)[:, :k]
    assert torch.equal(got_steps.cpu(), steps.abs())
    assert torch.equal(got_zeros.cpu(), torch.where(negative, 15 - zeros, zeros))
    assert torch.equal(ops.unpack_int4(packed, k).cpu(), torch.where(by_column, 15 - codes, codes))


@pytest.mark.parametrize("route,m,n,k", [(_native.ROUTE_TILE, 8, 100, 520), (_native.ROUTE_STREAM, 8, 1000, 520), (_native.ROUTE_STREAM, 40, 300, 257),
                                         (_native.ROUTE_BATCH, 64, 300, 520), (_native.ROUTE_TCGEN05, 256, 304, 520)])
def test_products_read_the_weights(route, m, n, k):
    codes, steps, zeros = _state(n, k)
    packed, steps, zeros = ops.pack_int4(codes.cuda()), steps.cuda(), zeros.cuda()
    image = _native.repack(packed, steps, zeros, k)
    weights = ops.dequantize_int4(packed, steps, zeros, k).half()
    for first in range(0, k, m):
        columns = torch.arange(first, min(first + m, k), device="cuda")
        x = torch.zeros(m, k, dtype=torch.float16, device="cuda")
        x[torch.arange(len(columns), device="cuda"), columns] = 1.0
        assert torch.equal(_native.linear(x, image, n, k, route=route)[: len(columns)], weights[:, columns].t())
    assert _native.status() == 0
