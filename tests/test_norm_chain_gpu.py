"""RmsNormLinear in a chain of programmatic dependents: the norm kernel signals the projection behind it before it waits for the
projection in front of it, so all three can be resident at once.  Each may read only what its predecessor has finished
writing: with B2_FLAG_OVERLAP_LAUNCH the chain must give the bits of ordinary launches.  Rows of up to 8192 columns stay in
the norm kernel's registers, longer ones are read back."""
import pytest
import torch

import dandan_ops_b200 as ops
from dandan_ops_b200 import _native
from oracle import w4a16_oracle as oracle

pytestmark = pytest.mark.gpu


def _layer(n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return ops.QuantizedLinear.from_float((torch.randn(n, k, generator=g, device="cuda") * 0.02).half())


def _chain(first, middle, last, weight, x0, other, role, flags, buffers):
    """first writes x or the residual of the norm in front of `middle`, whose output is the x of `last`."""
    mid, end = buffers
    _native.linear(x0, first._native_image(), first.out_features, first.in_features, out=mid, flags=flags)
    x, residual = (mid, other) if role == "x" else (other, mid)
    y, summed = _native.rmsnorm_linear(x, residual, weight, 1e-6, middle._native_image(), middle.out_features, middle.in_features, flags=flags)
    _native.linear(y, last._native_image(), last.out_features, last.in_features, out=end, flags=flags)
    return mid, y, summed, end


@pytest.mark.parametrize("k", [1024, 8192, 8200, 9216])
@pytest.mark.parametrize("m", [1, 8, 16, 40, 200])
@pytest.mark.parametrize("role", ["x", "residual"])
def test_norm_between_two_projections(role, m, k):
    first, middle, last = _layer(k, 1024, 1), _layer(1024, k, 2), _layer(2048, 1024, 3)
    g = torch.Generator().manual_seed(m + k)
    x0, other = torch.randn(m, 1024, generator=g).half().cuda(), torch.randn(m, k, generator=g).half().cuda()
    weight = (1.0 + 0.1 * torch.randn(k, generator=g)).half().cuda()
    buffers = [torch.empty(m, k, dtype=torch.float16, device="cuda"), torch.empty(m, 2048, dtype=torch.float16, device="cuda")]

    def run(flags):
        return _chain(first, middle, last, weight, x0, other, role, flags, buffers)

    want = [t.clone() for t in run(0)]
    for _ in range(3):
        for t in buffers:
            t.fill_(float("nan"))
        got = run(_native.FLAG_OVERLAP_LAUNCH)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with _native.private_workspace(), torch.cuda.graph(graph, stream=stream):
            got = [run(_native.FLAG_OVERLAP_LAUNCH) for _ in range(2)][-1]
        for _ in range(3):
            for t in buffers:
                t.fill_(float("nan"))
            graph.replay()
            stream.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    del graph
    assert _native.status() == 0


def test_norm_behind_a_copy_in_a_graph():
    """The module as the first kernel behind a memcpy node, which cannot be overlapped."""
    norm = ops.RmsNormLinear(torch.ones(2048, device="cuda"), _layer(1024, 2048, 5), eps=1e-6)
    static, new = (torch.randn(4, 2048, generator=torch.Generator().manual_seed(s)).half().cuda() for s in (1, 2))
    want = [t.clone() for t in norm(new)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        norm(static)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            static.copy_(new)
            got = norm(static)
        graph.replay()
        stream.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    del graph


@pytest.mark.parametrize("k", [8184, 8192, 8200, 16384, 16392, 28672])
@pytest.mark.parametrize("with_residual,want_sum", [(True, True), (True, False), (False, True)])
def test_long_rows_against_the_oracle(with_residual, want_sum, k):
    g = torch.Generator().manual_seed(k)
    x, residual = torch.randn(3, k, generator=g).half(), torch.randn(3, k, generator=g).half()
    weight = (1.0 + 0.1 * torch.randn(k, generator=g)).half()
    ref, ref_sum = oracle.residual_rms_norm(x.numpy(), (residual if with_residual else torch.zeros_like(x)).numpy(), weight.numpy(), 1e-6)
    out, summed = _native.residual_rms_norm(x.cuda(), residual.cuda() if with_residual else None, weight.cuda(), 1e-6, want_sum=want_sum)
    if want_sum:
        assert torch.equal(summed.cpu(), torch.from_numpy(ref_sum))
    # another order of the FP32 sum of squares moves the mean by a few 2^-24: a value may round to its FP16 neighbour
    # (2^-10 of it), and the product with the weight once more
    torch.testing.assert_close(out.cpu(), torch.from_numpy(ref), atol=1e-6, rtol=2.0 ** -9)
    assert float((out.cpu() != torch.from_numpy(ref)).float().mean()) < 5e-3
