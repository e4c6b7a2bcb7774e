"""One-pass quantizer and dequantizer on the GPU against the oracle, at the edges of their words, groups and blocks."""
import numpy as np
import pytest
import torch

import cases
import dandan_ops_b200 as ops
from dandan_ops_b200 import _native
from oracle import w4a16_oracle as oracle

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (3, 7), (16, 64), (17, 65), (15, 255), (33, 257), (40, 520), (129, 1000), (64, 2048)]


def weights(n, k, kind, dtype):
    g = torch.Generator().manual_seed(n * 1009 + k)
    w = torch.randn(n, k, generator=g)
    if kind == "grid":                       # quotients on and next to half-integers
        w = torch.randint(-30, 31, (n, k), generator=g).float() * 0.5
        w[:, ::64] = -7.5
        w[:, 1::64] = 7.5
    elif kind == "wide":                     # steps from the smallest normal number to beyond 2^100
        w = w * (10.0 ** torch.randint(-39, 37, (n, 1), generator=g).double()).float()
    elif kind == "positive":
        w = w.abs()
        w[0] = 0.0
    return w.to(dtype)


@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("kind,dtype", [("gauss", torch.float16), ("gauss", torch.float32), ("grid", torch.float16),
                                        ("wide", torch.float32), ("positive", torch.float16)])
def test_quantizer_is_the_oracle_bit_for_bit(n, k, kind, dtype):
    w = weights(n, k, kind, dtype)
    codes, steps, zeros = oracle.quantize(w.numpy())
    got = [t.cpu().numpy() for t in ops.quantize_int4(w.cuda())]
    assert np.array_equal(got[0], codes) and np.array_equal(got[2], zeros)
    assert np.array_equal(got[1].view(np.uint32), steps.view(np.uint32))
    layer = ops.QuantizedLinear.from_float(w.cuda())
    assert np.array_equal(layer.packed_weight.cpu().numpy(), oracle.pack(codes))
    assert torch.equal(layer._native_image(), _native.repack(layer.packed_weight, layer.scales, layer.zeros, k))
    assert layer._image_flags == layer._layer_flags()
    # an unaligned weight takes the element-wise loads
    shifted = torch.empty(n * k + 1, dtype=dtype, device="cuda")[1:].view(n, k)
    shifted.copy_(w)
    again = ops.QuantizedLinear.from_float(shifted)
    assert torch.equal(again._native_image(), layer._native_image()) and torch.equal(again.packed_weight, layer.packed_weight)


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("at", [(0, 0), (16, 256), (16, 128)])
def test_quantizer_rejects_a_single_nonfinite_weight(bad, at):
    w = torch.randn(17, 257)
    w[at] = bad
    with pytest.raises(ValueError, match="finite"):
        ops.QuantizedLinear.from_float(w.cuda())


@pytest.mark.parametrize("n,k", SHAPES)
def test_dequantizers_are_the_oracle_bit_for_bit(n, k):
    words, steps, zeros = cases.direct_state(n, k, n + k, lambda c: ops.pack_int4(c.cuda()))
    want = oracle.dequantize(words.cpu().numpy(), steps.numpy(), zeros.numpy(), k)
    got = ops.dequantize_int4(words, steps.cuda(), zeros.cuda(), k)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
    image = _native.repack(words, steps.cuda(), zeros.cuda(), k)
    assert torch.equal(_native.dequantize(image, n, k), got)
    assert torch.equal(_native.dequantize(image, n, k, torch.float16), got.half())
