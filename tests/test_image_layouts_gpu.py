"""Image files from before there were factored steps (layout 1): read, and their steps brought to the form that decodes fastest."""
import struct
import zlib

import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native, checkpoint

pytestmark = pytest.mark.gpu


def _plain(image, scales, n, k):
    """The image as layout 1 has it: the FP32 step of every group, 1 where there is none."""
    steps = torch.ones(-(-n // 16) * 16, -(-k // 256) * 4)
    steps[:n, : scales.shape[1]] = scales.cpu()
    by_block = steps.view(-1, 2, 8, steps.shape[1] // 4, 4).permute(3, 0, 2, 4, 1).reshape(-1, 64)
    blocks = image.cpu().clone().view(-1, 2336)
    blocks[:, 2048:2304] = by_block.contiguous().view(torch.uint8)
    return blocks.reshape(-1)


@pytest.mark.parametrize("n,k", [(100, 520), (256, 1024)])
def test_a_file_of_layout_1(tmp_path, n, k):
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=torch.Generator().manual_seed(n)) * 0.02).half().cuda())
    old = _plain(layer._native_image(), layer.scales, n, k).numpy()
    x = torch.randn(4, k, generator=torch.Generator().manual_seed(2)).half().cuda()
    plain = torch.from_numpy(old).cuda()
    assert torch.equal(_native.linear(x, plain, n, k), layer(x))                 # read by the kernels as it is
    cache = checkpoint.ImageCache(tmp_path)
    with open(cache.path_for(layer), "wb") as f:
        f.write(struct.Struct("<8sIIqqqI20x").pack(checkpoint.IMAGE_MAGIC, 1, 2, n, k, old.size, zlib.crc32(old.tobytes())))
        f.write(old.tobytes())
    state = {key: v.cpu() if isinstance(v, torch.Tensor) else v for key, v in layer.state_dict().items()}
    again, hit = cache.load_layer(state)
    assert hit and again._image_flags == layer._image_flags
    twin = ops.QuantizedLinear(layer.packed_weight, layer.scales, layer.zeros, in_features=k)
    assert cache.attach(twin)
    for got in (again, twin):
        fields = [i._native_image().view(-1, 2336)[:, 2048:2304].contiguous().view(torch.int32) for i in (got, layer)]
        real = fields[1] != fields[1][-1, -1] if n % 16 else torch.ones_like(fields[1], dtype=torch.bool)      # (padding had a step of 1)
        assert torch.equal(fields[0][real], fields[1][real]) and (fields[0] < 0).float().mean() > 0.99
        assert torch.equal(got(x), layer(x))


@pytest.mark.parametrize("n,k", [(100, 520), (256, 1024)])
@pytest.mark.parametrize("sigma,flag", [(0.02, 0), (2e-4, _native.FLAG_PLAIN_STEPS)])
@pytest.mark.parametrize("layout", [1, 2])
def test_flags_of_a_layer_from_a_file(tmp_path, layout, sigma, flag, n, k):
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=torch.Generator().manual_seed(n)) * sigma).half().cuda())
    assert layer._image_flags & _native.FLAG_PLAIN_STEPS == flag
    cache = checkpoint.ImageCache(tmp_path)
    path = cache.store(layer)
    if layout == 1:
        data = _plain(layer._native_image(), layer.scales, n, k).numpy().tobytes()
        with open(path, "wb") as f:
            f.write(struct.Struct("<8sIIqqqI20x").pack(checkpoint.IMAGE_MAGIC, 1, 2, n, k, len(data), zlib.crc32(data)) + data)
    again, hit = cache.load_layer({key: v.cpu() if isinstance(v, torch.Tensor) else v for key, v in layer.state_dict().items()})
    assert hit and again._image_flags == layer._image_flags == again._layer_flags()
    x = torch.randn(4, k, generator=torch.Generator().manual_seed(2)).half().cuda()
    assert torch.equal(again(x), layer(x))
