"""What a layer derives from its tensors (the image, the FP16 bias) belongs to those tensors: others that turn up at the same address, with the
same version, get their own."""
import copy
import ctypes
import pickle

import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native


class _Memory:
    """Memory that any number of tensors, each with a version counter of its own, are made over."""

    def __init__(self, like):
        self.held = like.clone()
        types = {torch.float32: "<f4", torch.int32: "<i4", torch.float16: "<f2"}
        self.__cuda_array_interface__ = {"shape": tuple(like.shape), "typestr": types[like.dtype], "data": (self.held.data_ptr(), False), "version": 3}

    def tensor(self):
        return torch.as_tensor(self, device="cuda")


def test_a_new_bias_at_the_address_of_the_old_one():
    data = (ctypes.c_float * 32)(*range(32))
    layer = ops.QuantizedLinear.from_float(torch.randn(32, 64))
    layer.bias = torch.frombuffer(data, dtype=torch.float32)
    assert torch.equal(layer._bias_fp16(), torch.arange(32).half())
    layer.bias = None
    for i in range(32):
        data[i] = -i
    layer.bias = torch.frombuffer(data, dtype=torch.float32)
    assert torch.equal(layer._bias_fp16(), -torch.arange(32).half())


def test_a_layer_can_be_copied_and_pickled():
    layer = ops.QuantizedLinear.from_float(torch.randn(32, 64), torch.randn(32))
    layer._bias_fp16()
    for other in (copy.deepcopy(layer), pickle.loads(pickle.dumps(layer))):
        assert torch.equal(other.packed_weight, layer.packed_weight) and torch.equal(other._bias_fp16(), layer._bias_fp16())
        assert other._bias16 is not layer._bias16


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["packed_weight", "scales", "zeros", "bias"])
def test_new_tensors_at_the_addresses_of_the_old_ones(which):
    g = torch.Generator(device="cuda").manual_seed(1)
    first, second = (ops.QuantizedLinear.from_float(torch.randn(64, 128, generator=g, device="cuda").half(), torch.randn(64, generator=g, device="cuda"))
                     for _ in range(2))
    x = torch.randn(3, 128, generator=g, device="cuda").half()
    memory = {name: _Memory(getattr(first, name)) for name in ("packed_weight", "scales", "zeros", "bias")}
    for name in memory:
        setattr(first, name, memory[name].tensor())
    want = first(x)
    assert torch.equal(first(x), want)
    setattr(first, which, None)
    memory[which].held.copy_(getattr(second, which))
    setattr(first, which, memory[which].tensor())
    fresh = ops.QuantizedLinear(*(t.clone() for t in (first.packed_weight, first.scales, first.zeros)), in_features=128, bias=first.bias.clone())
    got = first(x)
    assert torch.equal(got, fresh(x)) and not torch.equal(got, want) and torch.equal(first(x), got)
    assert torch.equal(first.forward_into(x, torch.empty_like(got)), got)


@pytest.mark.gpu
def test_a_state_that_comes_back():
    """Another state in between, seen only by the raw entry point, leaves no image of its own behind."""
    g = torch.Generator(device="cuda").manual_seed(2)
    layer, other = (ops.QuantizedLinear.from_float(torch.randn(64, 128, generator=g, device="cuda").half()) for _ in range(2))
    x = torch.randn(3, 128, generator=g, device="cuda").half()
    want, out = layer(x), torch.empty(3, 64, dtype=torch.float16, device="cuda")
    layer(x)
    kept = layer.scales
    layer.scales = other.scales
    assert not torch.equal(layer.forward_into(x, out), want)
    layer.scales = kept
    assert torch.equal(layer(x), want)


@pytest.mark.gpu
@pytest.mark.parametrize("operator", [False, True])
def test_state_by_value_with_temporary_scales(operator):
    """Temporaries of one size follow each other at one address, given to the functional form and to the operators of the reference."""
    g = torch.Generator(device="cuda").manual_seed(3)
    layer = ops.QuantizedLinear.from_float(torch.randn(64, 128, generator=g, device="cuda").half())
    x = torch.randn(3, 128, generator=g, device="cuda").half()

    def call(factor):
        if operator:
            return torch.ops.dandan_ops.w4a16_tensorcore(x, layer.packed_weight, layer.scales * factor, layer.zeros, 64)
        return ops.quantized_linear(x, layer.packed_weight, layer.scales * factor, layer.zeros, in_features=128)

    once = call(1.0)
    assert torch.equal(call(2.0), once * 2) and torch.equal(call(1.0), once)


@pytest.mark.gpu
def test_what_is_known_of_an_image_comes_with_it(monkeypatch):
    """A read of the new image's steps that fails leaves no image behind that runs under the old one's flags."""
    g = torch.Generator(device="cuda").manual_seed(4)
    layer = ops.QuantizedLinear.from_float(torch.randn(64, 128, generator=g, device="cuda").half())
    x = torch.randn(3, 128, generator=g, device="cuda").half()
    want, steps = layer(x), layer.scales
    layer.scales = steps.half().float()
    layer(x)
    assert layer._image_flags & _native.FLAG_FP16_STEPS
    layer.scales = steps

    def fails(*args):
        raise RuntimeError("read")

    with monkeypatch.context() as patch:
        patch.setattr(_native, "image_flags", fails)
        with pytest.raises(RuntimeError, match="read"):
            layer(x)
    assert torch.equal(layer(x), want) and not layer._image_flags & _native.FLAG_FP16_STEPS
