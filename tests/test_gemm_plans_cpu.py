"""CTAs along K that the shape model of the pair GEMM chooses, where the measured times of the choices differ by 4 % or more."""
import pytest

from dandan_ops_b200 import _native


@pytest.mark.parametrize("m,n,k,splits", [
    (200, 6144, 4096, 3), (256, 6144, 4096, 3), (384, 6144, 4096, 3), (512, 6144, 4096, 1), (512, 3072, 4096, 3), (768, 3072, 4096, 2),
    (1536, 1024, 3072, 3), (2048, 1024, 3072, 2), (3072, 1024, 3072, 1), (1024, 4096, 12288, 1), (768, 4096, 4096, 1),
    (384, 4096, 4096, 2), (2048, 8192, 28672, 2)])
def test_splits(m, n, k, splits):
    assert _native.plan(m, n, k)["k_splits"] == splits
