"""The tile kernel with two row tiles per CTA beside the form with one (which an x that is not aligned takes): the same bits, and gate/up pairs
on shapes that the plan gives to this form."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu
TILE = _native.ROUTE_TILE


def _layer(n, k, seed, kind="mixed"):
    g = torch.Generator(device="cuda").manual_seed(seed)
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * (0.0006 if kind == "plain" else 0.02)).half())
    if kind == "fp16":
        layer = ops.QuantizedLinear(layer.packed_weight, layer.scales.half().float(), layer.zeros, in_features=k)
    return layer, g


def _takes_two_tiles(m, n, k):
    """What tile_pair_applicable() asks of an aligned x, and what the plan says where the automatic route takes the tile kernel."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 8 < m <= 16 and sms < -(-n // 16) <= 2 * sms and k > 1792 and k % 8 == 0
    plan = _native.plan(m, n, k)
    if plan["route"] == "b200_tile":
        assert plan["grid"] == (-(-n // 16) + 1) // 2
    return plan["route"] == "b200_tile"


def _misaligned(x):
    out = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)[1:].view(x.shape)
    return out.copy_(x)


@pytest.mark.parametrize("m,n,k,kind", [(9, 2384, 2048, "mixed"), (16, 4736, 2048, "mixed"), (16, 2385, 1800, "plain"), (12, 3840, 4352, "mixed"),
                                        (10, 3828, 4104, "fp16"), (15, 3000, 3080, "plain"), (16, 4096, 4096, "fp16")])
def test_the_bits_of_one_tile_per_cta(m, n, k, kind):
    layer, g = _layer(n, k, n + k, kind)
    image, flags = layer._native_image(), layer._image_flags
    _takes_two_tiles(m, n, k)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    assert torch.equal(_native.linear(_misaligned(x), image, n, k, route=TILE, flags=flags), _native.linear(x, image, n, k, route=TILE, flags=flags))


@pytest.mark.parametrize("m,n,k", [(11, 4000, 2048), (9, 2416, 1800), (16, 4096, 4096), (13, 3600, 4104)])
def test_gate_up_pairs(m, n, k):
    assert _takes_two_tiles(m, n, k)                       # (the fused call has the automatic route only)
    layer, g = _layer(n, k, 3)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    lib, out = _native.load(), torch.zeros(m, n // 2, dtype=torch.float16, device="cuda")
    big = _native.linear(_misaligned(x), layer._native_image(), n, k, route=TILE)
    ws = torch.zeros(int(lib.b2_w4a16_workspace_bytes(m, n, k)), dtype=torch.uint8, device="cuda")
    assert lib.b2_w4a16_linear_silu_mul(x.data_ptr(), k, layer._native_image().data_ptr(), None, out.data_ptr(), n // 2, m, n, k, ws.data_ptr(),
                                        ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, _native.silu_mul_pairs(big))
