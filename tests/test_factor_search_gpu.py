"""The search for factored step fields (csrc/factor_steps.cuh): every field that it writes gives the sixteen weights of its group by
the operations of the factored chain, and few groups are left without one."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native

pytestmark = pytest.mark.gpu


def _fields(image):
    blocks = image.view(-1, 2336)
    z = blocks[:, 2304:2336]
    zeros = torch.stack([z & 15, z >> 4], dim=2).reshape(-1, 64).int()
    return blocks[:, 2048:2304].contiguous().view(torch.int32), zeros


def _check_fields(image):
    """The factored chain in FP32 arithmetic rounded to FP16 after each operation: products and sums of FP16 numbers with these few
    significant bits are exact in FP32, so each rounding is the instruction's own."""
    fields, zeros = _fields(image)
    mask = fields < 0
    f, z = fields[mask].long() & 0xFFFFFFFF, zeros[mask]
    a1 = 1.0 + (f >> 3 & 127).float() / 128
    a2 = (f >> 16 & 0x3FFF | 0x4000).to(torch.int16).view(torch.float16).float()
    b = (-(z.float() * a1) * 2.0 ** -14).half().float()
    remainder = ((f >> 30 & 1) << 9 | (f >> 10 & 63) << 3 | f & 7) - 512
    step = ((a1 * a2 * 2.0 ** -14).view(torch.int32) + remainder.int()).view(torch.float32)
    for code in range(16):
        first = (code * a1 * 2.0 ** -14 + b).half().float()
        got = (first * a2).half()
        want = ((code - z).float() * step).half()
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), code
    return mask


# (groups without factors in 10^4, blocks with a factored field for every group in 100): measured 0.3 / 23 / 119 / 224 and
# 99.8 / 86 / 46 / 23 on 786432 groups
@pytest.mark.parametrize("n,k", [(1000, 520), (1024, 4096), (4096, 12288)])
@pytest.mark.parametrize("kind,plain,whole", [("fp16", 3, 95), ("fp32", 50, 70), ("positive fp16", 200, 25), ("negative fp16", 250, 15),
                                              ("positive fp32", 350, 8)])
def test_fields_and_their_share(kind, plain, whole, n, k):
    w = torch.randn(n, k, generator=torch.Generator(device="cuda").manual_seed(n + k), device="cuda") * 0.02
    w = w.abs() if "positive" in kind else -w.abs() if "negative" in kind else w
    layer = ops.QuantizedLinear.from_float(w.half() if "fp16" in kind else w)
    mask = _check_fields(layer._native_image())
    assert (~mask).float().mean() * 1e4 < plain and mask.all(1).float().mean() * 100 > whole
    assert torch.equal(layer._native_image(), _native.repack(layer.packed_weight, layer.scales, layer.zeros, k))
    for got, want in zip(_native.unrepack(layer._native_image(), n, k), (layer.packed_weight, layer.scales, layer.zeros)):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))


def test_every_zero_point_and_the_whole_range():
    n, k = 2048, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    codes = torch.randint(0, 16, (n, k), generator=g, dtype=torch.uint8, device="cuda")
    zeros = torch.randint(0, 16, (n, k // 64), generator=g, dtype=torch.int32, device="cuda")
    steps = torch.exp2(-12 + 13.9 * torch.rand(n, k // 64, generator=g, device="cuda"))
    image = _native.repack(ops.pack_int4(codes), steps, zeros, k)
    assert _check_fields(image).float().mean() > 0.95
    got = _native.unrepack(image, n, k)
    assert torch.equal(got[1].view(torch.int32), steps.view(torch.int32)) and torch.equal(got[2], zeros)
    # once more over its own fields: nothing changes
    again = image.clone()
    _native.factor_steps(again, n, k)
    assert torch.equal(again, image)


@pytest.mark.parametrize("n,k", [(64, 256), (1000, 520)])
def test_steps_outside_the_range_stay_plain(n, k):
    w = torch.randn(n, k, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * 2e-4
    layer = ops.QuantizedLinear.from_float(w)
    fields, _ = _fields(layer._native_image())
    padding = torch.zeros(-(-n // 16) * 16, -(-k // 256) * 4, dtype=torch.bool)
    padding[n:] = True
    padding[:, -(-k // 64):] = True
    by_block = padding.view(-1, 2, 8, padding.shape[1] // 4, 4).permute(3, 0, 2, 4, 1).reshape(-1, 64)       # field: row g + 8h, group t -> (g, t, h)
    assert torch.equal(fields.cpu() < 0, by_block)


def test_a_converted_layer_is_complete():
    """Nothing of the conversion is still running when the layer is returned: the image may be read on any stream."""
    w = (torch.randn(28672, 4096, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") * 0.02).half()
    for _ in range(3):
        layer = ops.QuantizedLinear.from_float(w)
        assert torch.cuda.current_stream().query()
        assert _native.FLAG_OVERLAP_LAUNCH & layer._image_flags or not _native.OVERLAP_LAUNCH
