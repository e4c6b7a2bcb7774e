"""w4a16_batch_kernel (up to 128 rows of x, products on tcgen05): against the CPU oracle and, on its other forms, against
the routes it stands in for, at the sizes where tiles, ranges and rings end."""
import ctypes

import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native
from oracle import w4a16_oracle as oracle

pytestmark = pytest.mark.gpu
BATCH = _native.ROUTE_BATCH


def _layer(n, k, seed, fp16_steps=False):
    g = torch.Generator().manual_seed(seed)
    layer = ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g) * 0.02).half().cuda())
    if fp16_steps:
        layer = ops.QuantizedLinear(layer.packed_weight, layer.scales.half().float(), layer.zeros, in_features=k)
    return layer, g


@pytest.mark.parametrize("m,n,k,fp16_steps", [
    (1, 8, 8, False),            # one partial tile, one partial step
    (16, 128, 256, False),       # one whole tile in one block, fewer steps than CTAs
    (17, 136, 1032, True),       # a second tile of one row tile, ragged K
    (32, 1000, 520, False),
    (33, 129, 64, False),        # one row in the last tile, one group of the block
    (64, 2048, 1024, True),      # tiles shared by several CTAs
    (65, 384, 8192, False),      # K much longer than a CTA's range
    (100, 1536, 2056, False),
    (128, 20000, 128, False),    # several one-block tiles per CTA
])
def test_against_the_oracle(m, n, k, fp16_steps):
    layer, g = _layer(n, k, m + n + k, fp16_steps)
    x = torch.randn(m, k, generator=g).half()
    bias = torch.randn(n, generator=g).half().cuda()
    image, flags = layer._native_image(), layer._image_flags
    assert bool(flags & _native.FLAG_FP16_STEPS) == fp16_steps
    y = _native.linear(x.cuda(), image, n, k, route=BATCH, flags=flags)
    assert torch.equal(y, _native.linear(x.cuda(), image, n, k, route=BATCH, flags=flags & ~_native.FLAG_OVERLAP_LAUNCH))
    assert torch.equal(y + bias, _native.linear(x.cuda(), image, n, k, route=BATCH, bias=bias, flags=flags))
    words, step, zero = (t.cpu().numpy() for t in (layer.packed_weight, layer.scales, layer.zeros))
    rows = sorted({0, m // 2, m - 1})                                    # (the oracle is slow)
    assert oracle.within_tolerance(y[rows].cpu().numpy(), oracle.linear(x[rows].numpy(), words, step, zero, k))
    # every row and column: FP64 product of the same FP16 weights, one FP16 rounding apart at most where sums round differently
    exact = x.double() @ layer.dequantize().half().double().cpu().t()
    assert ((y.cpu().double() - exact).abs() <= 2e-3 + 2e-3 * exact.abs()).all()
    assert _native.status() == 0


def test_row_strides_of_x_and_y():
    layer, g = _layer(1000, 520, 5)
    wide = torch.randn(48, 536, generator=g).half().cuda()
    out = torch.full((48, 1010), 7.0, dtype=torch.float16, device="cuda")
    want = _native.linear(wide[:, 8:528].contiguous(), layer._native_image(), 1000, 520, route=BATCH)
    _native.linear(wide[:, 8:528], layer._native_image(), 1000, 520, route=BATCH, out=out[:, 3:1003])
    assert torch.equal(out[:, 3:1003], want) and bool((out[:, :3] == 7).all()) and bool((out[:, 1003:] == 7).all())


@pytest.mark.parametrize("m,rows,k", [(33, 72, 264), (64, 1536, 1024), (1, 4096, 2304), (12, 32768, 520), (128, 32768, 1032)])
def test_gate_up_epilogue_matches_the_separate_kernel(m, rows, k):
    """The automatic route takes the batch kernel on these; the activation sees the same sums in the same order."""
    gate, g = _layer(rows, k, 1)
    up, _ = _layer(rows, k, 2)
    fused = ops.GateUpSilu(gate, up)
    x = torch.randn(m, k, generator=g).half().cuda()
    pairs = _native.linear(x, fused.op._native_image(), 2 * rows, k, route=BATCH)
    assert torch.equal(fused(x), _native.silu_mul_pairs(pairs))


def test_dependent_launches_on_shared_scratch():
    """Programmatic dependents: every call reads the previous one's output and shares its tickets and partial tiles."""
    layers = [_layer(2048, 2048, s)[0] for s in range(5)]
    x = torch.randn(40, 2048, generator=torch.Generator().manual_seed(9)).half().cuda()

    def chain(flags):
        cur = x
        for layer in layers:
            cur = _native.linear(cur, layer._native_image(), 2048, 2048, route=BATCH, flags=flags)
        return cur

    want = chain(0)
    for _ in range(10):
        assert torch.equal(chain(_native.FLAG_OVERLAP_LAUNCH), want)


def test_what_the_route_refuses():
    layer, _ = _layer(64, 520, 3)
    x = torch.zeros(129, 520, dtype=torch.float16, device="cuda")
    with pytest.raises(RuntimeError, match="batch route"):
        _native.linear(x, layer._native_image(), 64, 520, route=BATCH)
    odd = torch.zeros(40 * 520 + 1, dtype=torch.float16, device="cuda")[1:].view(40, 520)      # not 16-byte aligned
    with pytest.raises(RuntimeError, match="batch route"):
        _native.linear(odd, layer._native_image(), 64, 520, route=BATCH)
    assert torch.equal(_native.linear(odd, layer._native_image(), 64, 520), torch.zeros(40, 64, dtype=torch.float16, device="cuda"))


@pytest.mark.parametrize("m,skipped", [(9, 0), (9, 5), (40, 1), (128, 3)])
def test_a_wait_that_runs_out_sets_the_status_word_and_returns(m, skipped):
    """One weight copy of the first CTA is left out: all roles give up, every copy and product in flight ends, and tensor
    memory is freed (the next call needs all of it)."""
    n, k = 4096, 8192
    layer, g = _layer(n, k, 77)
    x = torch.randn(m, k, generator=g).half().cuda()
    lib, image = _native.load(), layer._native_image()
    ws = torch.zeros(int(lib.b2_w4a16_workspace_bytes(m, n, k)), dtype=torch.uint8, device="cuda")
    word = ctypes.c_uint(7)

    def call():
        y = torch.zeros(m, n, dtype=torch.float16, device="cuda")
        assert lib.b2_w4a16_linear_route(x.data_ptr(), k, image.data_ptr(), y.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(),
                                         torch.cuda.current_stream().cuda_stream, BATCH) == 0
        assert lib.b2_w4a16_status(ws.data_ptr(), None, ctypes.byref(word)) == 0
        return y

    good = call()
    assert word.value == 0
    _native.test_hooks(wait_limit=64, skip_copy=skipped)
    try:
        call()
        assert word.value == 2
    finally:
        _native.test_hooks()
    ws.zero_()
    assert torch.equal(call(), good) and word.value == 0


@pytest.mark.parametrize("m,n,k", [(16, 4096, 8192), (128, 2048, 2048), (40, 256, 256)])
def test_the_wait_limit_does_not_count_the_kernel_before(m, n, k):
    """A dependent launch beside a predecessor that lasts longer than the poll limit: a one-launch gather of a small slice,
    most SMs left free, that waits 0.2 s for packets that never arrive."""
    layer, g = _layer(n, k, 5)
    x = torch.randn(m, k, generator=g).half().cuda()
    image = layer._native_image()
    want = _native.linear(x, image, n, k, route=BATCH, flags=layer._image_flags)
    piece, _ = _layer(32, 1032, 6)
    bufs = [torch.zeros(1, 64, dtype=torch.float16, device="cuda") for _ in range(2)]
    boxes = [torch.zeros(_native.gather_block_bytes(2, 4096), dtype=torch.uint8, device="cuda") for _ in range(2)]
    one = torch.randn(1, 1032, generator=g).half().cuda()
    assert _native.linear_gather_launches(1, 64, 32, 1032, 0, 2, 4096) == 1
    torch.cuda.synchronize()
    _native.gather_wait_limit(200000)
    _native.test_hooks(wait_limit=64)                                    # about a millisecond
    try:
        _native.linear_gather(one, piece._native_image(), 1032, [t.data_ptr() for t in bufs], [t.data_ptr() for t in boxes], 4096, 0,
                              64, 64, 32)
        y = _native.linear(x, image, n, k, route=BATCH, flags=_native.FLAG_OVERLAP_LAUNCH)
        torch.cuda.synchronize()
    finally:
        _native.gather_wait_limit(0)
        _native.test_hooks()
    assert _native.gather_status(boxes[0].data_ptr()) & 4                # the predecessor did wait until its own limit
    assert torch.equal(y, want) and _native.status() == 0


def _not_nearest(y, exact):
    """Share of FP16 outputs that are not the nearest to the 64-bit sum: proportional to the error of the FP32 sums."""
    return float((y != exact.to(torch.float16)).double().mean())


@pytest.mark.parametrize("m,n,k,replaced", [
    (9, 6144, 4096, _native.ROUTE_STREAM),
    (16, 4096, 12288, _native.ROUTE_STREAM),
    (24, 6144, 4096, _native.ROUTE_STREAM),
    (32, 4096, 12288, _native.ROUTE_STREAM),
    (64, 4096, 12288, _native.ROUTE_TCGEN05),
    (128, 8192, 4096, _native.ROUTE_TCGEN05),
])
def test_sums_are_no_further_off_than_those_of_the_kernel_it_replaces(m, n, k, replaced):
    """Against 64-bit sums, over every output.  The bound allows a tenth more, and four standard deviations of the count."""
    layer, g = _layer(n, k, 3)
    x = torch.randn(m, k, generator=g).half().cuda()
    image = layer._native_image()
    exact = x.double() @ layer.dequantize().half().double().t()
    mine, theirs = (_not_nearest(_native.linear(x, image, n, k, route=r), exact) for r in (BATCH, replaced))
    assert mine <= 1.1 * theirs + 4 * (theirs / (m * n)) ** 0.5


def _raw(x, layer, ws_bytes, act=False):
    lib, (m, k), n = _native.load(), x.shape, layer.out_features
    ws = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda")
    y = torch.zeros(m, n // 2 if act else n, dtype=torch.float16, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    args = (x.data_ptr(), k, layer._native_image().data_ptr(), None, y.data_ptr(), y.stride(0), m, n, k, ws.data_ptr(), ws_bytes, stream)
    rc = lib.b2_w4a16_linear_silu_mul(*args) if act else lib.b2_w4a16_linear_bias(*args, _native.ROUTE_AUTO)
    assert rc == 0, lib.b2_w4a16_last_error()
    return y


@pytest.mark.parametrize("m,n,k", [(100, 6144, 4096), (128, 4096, 12288), (65, 1024, 8192)])
def test_one_workspace_for_all_batches(m, n, k):
    layer, g = _layer(n, k, 8)
    x = torch.randn(m, k, generator=g).half().cuda()
    size = _native.load().b2_w4a16_workspace_bytes
    want = _native.linear(x, layer._native_image(), n, k, route=BATCH)
    for larger in (m, 129, 256, 2048):
        assert torch.equal(_raw(x, layer, int(size(larger, n, k))), want)


def test_a_fused_call_runs_in_less_workspace_too():
    """What b2_w4a16_silu_mul_is_fused() promises does not depend on the workspace, nor on the GEMM's tile shape (the
    single-CTA ones, which a device without two-CTA clusters takes, have no such epilogue)."""
    m, n, k = 100, 512, 256
    layer, g = _layer(n, k, 8)
    x = torch.randn(m, k, generator=g).half().cuda()
    _native.set_gemm_shape("128x128")
    try:
        lib = _native.load()
        assert lib.b2_w4a16_silu_mul_is_fused(m, n, k)
        need = int(lib.b2_w4a16_workspace_bytes(m, n, k))
        torch.testing.assert_close(_raw(x, layer, need - 4096, act=True), _raw(x, layer, need, act=True), atol=2e-3, rtol=2e-3)
    finally:
        _native.set_gemm_shape()


@pytest.mark.parametrize("m,n,k,bad", [(9, 1000, 520, 4), (33, 384, 1032, 32), (70, 136, 264, 69)])
def test_a_row_that_is_not_finite_touches_no_other(m, n, k, bad):
    """Rows of x beyond M and weight rows beyond N are multiplied too: a NaN or an infinity stays in its row, and there is
    what an exact sum gives."""
    layer, g = _layer(n, k, 12)
    x = torch.randn(m, k, generator=g).half()
    image = layer._native_image()
    clean = _native.linear(x.cuda(), image, n, k, route=BATCH)
    x[bad, k - 1] = float("inf")
    x[bad, 3] = -float("inf")
    exact = x.double() @ layer.dequantize().half().double().cpu().t()
    y = _native.linear(x.cuda(), image, n, k, route=BATCH).cpu()
    others = [r for r in range(m) if r != bad]
    assert torch.equal(y[others], clean.cpu()[others])
    assert torch.equal(y[bad].isnan(), exact[bad].isnan()) and torch.equal(y[bad].isposinf(), exact[bad].isposinf())
    assert bool((y[bad].isnan() | y[bad].isinf()).all()) and bool(y[bad].isnan().any()) and bool(y[bad].isinf().any())
    x[bad, 5] = float("nan")
    y = _native.linear(x.cuda(), image, n, k, route=BATCH).cpu()
    assert torch.equal(y[others], clean.cpu()[others]) and bool(y[bad].isnan().all())
