"""dequantize_int4 at the edges of its runs of 256 columns: ragged last word, group and run, rows that are not 16-byte aligned, warps whose
runs cross rows, and one run in all; zero points beyond four bits as the image holds them, and a step that is not finite."""
import numpy as np
import pytest
import torch

from dandan_ops_b200 import _native
from oracle import w4a16_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (1, 256), (3, 257), (5, 4), (7, 252), (33, 260), (2, 1020), (9, 1021), (130, 68), (31, 516), (1000, 2308)])
def test_runs_of_256_columns(n, k):
    g = torch.Generator().manual_seed(n + k)
    groups = -(-k // 64)
    packed = torch.randint(-2**31, 2**31, (n, -(-k // 8)), generator=g).to(torch.int32)
    steps = torch.exp(torch.randn(n, groups, generator=g) * 3)
    steps[0, 0], steps[-1, -1] = float("inf"), -1e-39
    zeros = torch.randint(0, 16, (n, groups), generator=g, dtype=torch.int32)
    got = _native.dequantize_state(packed.cuda(), steps.cuda(), zeros.cuda() + 16, k).cpu().numpy()
    with np.errstate(all="ignore"):
        want = oracle.dequantize(packed.numpy(), steps.numpy(), zeros.numpy(), k)
    assert got.shape == want.shape and np.array_equal(got.view(np.uint32)[~np.isnan(want)], want.view(np.uint32)[~np.isnan(want)])
    assert np.array_equal(np.isnan(got), np.isnan(want))
