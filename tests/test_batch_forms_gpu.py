"""The work splits of w4a16_batch_kernel.  A cluster of CTAs per tile, whose sums meet in shared memory: every cluster size and
number of rows of x at the edges of its units of four columns, with K that does not divide evenly and a last tile that is not
whole.  Rounds of whole tiles: with none, one and many left over, shared by one CTA and by several.  Ranges where both leave SMs idle."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,act", [
    (16, 18944, 264, False), (9, 18952, 8200, False), (128, 19008, 4104, True), (33, 28672, 1032, False), (64, 24576, 2064, True),
    (17, 38400, 776, True), (16, 56848, 264, True), (128, 37900, 520, False), (16, 12304, 264, True), (40, 6160, 28680, False),
    (1, 8192, 4096, False), (5, 6144, 4104, True), (4, 5120, 5120, False), (13, 4097, 5000, False), (16, 1024, 3080, True),
    (17, 1000, 1544, False), (24, 5008, 5128, True), (32, 512, 8192, False), (33, 304, 2056, True), (61, 256, 8192, False),
    (64, 6144, 2048, False), (65, 129, 8200, False), (100, 5001, 5128, False), (128, 1024, 2304, True), (126, 7680, 2056, False)])
def test_against_64_bit_sums(m, n, k, act):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * 0.02).half())
    x = torch.randn(m, k, generator=g, device="cuda").half()
    bias = torch.randn(n, generator=g, device="cuda").half()
    image, flags = layer._native_image(), layer._image_flags
    y = _native.linear(x, image, n, k, route=_native.ROUTE_BATCH, flags=flags)
    # FP32 sums of at most K products and one rounding to FP16 (2^-11); the tensor core truncates, which the floor covers
    exact = x.double() @ layer.dequantize().half().double().t()
    assert ((y.double() - exact).abs() <= 2.0 ** -10 * exact.abs() + 2e-4).all()
    for _ in range(5):                                                       # neither timing nor the launch attribute shows
        assert torch.equal(_native.linear(x, image, n, k, route=_native.ROUTE_BATCH, flags=flags), y)
    assert torch.equal(_native.linear(x, image, n, k, route=_native.ROUTE_BATCH), y)
    assert torch.equal(_native.linear(x, image, n, k, route=_native.ROUTE_BATCH, bias=bias), y + bias)
    if act:                                                                  # the rows of the layer taken as gate/up pairs
        lib, out = _native.load(), torch.zeros(m, n // 2, dtype=torch.float16, device="cuda")
        ws = torch.zeros(int(lib.b2_w4a16_workspace_bytes(m, n, k)), dtype=torch.uint8, device="cuda")
        if _native.plan(m, n, k)["route"] == "b200_batch":
            assert lib.b2_w4a16_linear_silu_mul(x.data_ptr(), k, image.data_ptr(), None, out.data_ptr(), n // 2, m, n, k, ws.data_ptr(),
                                                ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
            assert torch.equal(out, _native.silu_mul_pairs(y))
    assert _native.status() == 0


@pytest.mark.parametrize("m,n,k,act", [
    (129, 1000, 520, False), (257, 1024, 2048, True), (512, 4096, 1032, False), (1024, 1024, 3080, True), (130, 6144, 2056, True),
    (1000, 128, 8200, False), (385, 2064, 264, True), (640, 3000, 3080, False), (1024, 2304, 776, False)])
def test_more_rows_than_one_tile_has(m, n, k, act):
    """The same splits over tiles of 128 rows of x, which the GEMM route takes for small layers: row tiles that are not whole, one CTA or
    a cluster per tile; the sums are those of the rows by themselves at the same split."""
    plan = _native.plan(m, n, k)
    assert plan["route"] == "b200_tcgen05" and plan["grid"] == -(-n // 128) * -(-m // 128) * plan["k_splits"]
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * 0.02).half())
    x = torch.randn(m, k, generator=g, device="cuda").half()
    wide = torch.randn(m, k + 8, generator=g, device="cuda").half()
    wide[:, :k] = x
    bias = torch.randn(n, generator=g, device="cuda").half()
    image, flags = layer._native_image(), layer._image_flags
    y = layer(x)
    exact = x.double() @ layer.dequantize().half().double().t()
    assert ((y.double() - exact).abs() <= 2.0 ** -10 * exact.abs() + 2e-4).all()          # (as above)
    assert torch.equal(_native.linear(wide[:, :k], image, n, k, route=_native.ROUTE_TCGEN05), y)
    out = torch.full((m, n + 6), 7.0, dtype=torch.float16, device="cuda")
    _native.linear(x, image, n, k, flags=flags, bias=bias, out=out[:, 3:n + 3])
    assert torch.equal(out[:, 3:n + 3], y + bias) and bool((out[:, :3] == 7).all()) and bool((out[:, n + 3:] == 7).all())
    if act:
        lib, half = _native.load(), torch.zeros(m, n // 2, dtype=torch.float16, device="cuda")
        ws = torch.zeros(int(lib.b2_w4a16_workspace_bytes(m, n, k)), dtype=torch.uint8, device="cuda")
        assert lib.b2_w4a16_silu_mul_is_fused(m, n, k)
        assert lib.b2_w4a16_linear_silu_mul(x.data_ptr(), k, image.data_ptr(), None, half.data_ptr(), n // 2, m, n, k, ws.data_ptr(),
                                            ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(half, _native.silu_mul_pairs(y))
    assert _native.status() == 0
