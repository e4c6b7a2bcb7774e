"""Errors of the FP32 sums, whichever kernel and split the automatic route takes: the share of FP16 outputs that are not the nearest to the
64-bit sum, over every output.  A tensor core drops the bits of a product below the running sum, so the share grows with the number of
products that one chain of sums takes.  Bounds: the tile kernel, whose chains have two to four products, where it takes the layer, else the
share (in per cent) of equal ranges of K with four chains up to 32 rows of x and two above, or of the two-SM GEMM above 128 rows,
measured with the same distributions.  Both with a tenth more, and four standard deviations of the counts."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu
TILE, AUTO = _native.ROUTE_TILE, _native.ROUTE_AUTO


@pytest.mark.parametrize("m,n,k,bound", [
    (8, 10240, 1536, TILE), (1, 12288, 1280, TILE), (8, 8192, 1280, TILE), (4, 6144, 2048, TILE), (8, 7168, 2048, TILE), (8, 4000, 4608, TILE),
    (8, 2048, 5120, TILE), (16, 8192, 1024, TILE), (16, 6144, 1024, TILE), (16, 5120, 1536, TILE), (16, 512, 8192, TILE), (9, 2048, 2048, TILE),
    (8, 24576, 4096, 0.60), (16, 24576, 4096, 0.434), (16, 28672, 1024, 0.141), (16, 16384, 8192, 0.705), (16, 8192, 1280, 0.119),
    (24, 6144, 4096, 0.214), (24, 2048, 5120, 0.124), (32, 28672, 4096, 0.440), (32, 5120, 1536, 0.105), (64, 6144, 4096, 0.373),
    (64, 5120, 1536, 0.172), (64, 28672, 1024, 0.244), (128, 6144, 4096, 0.372), (128, 24576, 4096, 0.775), (128, 2560, 9728, 0.385),
    (512, 3072, 3072, 0.530), (1024, 1536, 6144, 0.960), (512, 2560, 4096, 0.670)])
def test_no_further_off(m, n, k, bound):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * 0.02).half())
    image, weight = layer._native_image(), layer.dequantize().half().double().t()
    off, base, total = 0, 0, 0
    for _ in range(max(1, min(24, 2_000_000 // (m * n)))):
        x = torch.randn(m, k, generator=g, device="cuda").half()
        nearest = (x.double() @ weight).half()
        off += int((_native.linear(x, image, n, k, route=AUTO) != nearest).sum())
        base += int((_native.linear(x, image, n, k, route=TILE) != nearest).sum()) if bound == TILE else 0
        total += nearest.numel()
    limit = base if bound == TILE else bound / 100 * total
    assert off <= 1.1 * limit + 4 * (2 * limit) ** 0.5
