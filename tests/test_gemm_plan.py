"""The choice of a kernel for a product (``gemm_plan``), which needs no GPU."""

import pytest

from torchure_b200 import ops

_C = ops.ext()
pytestmark = pytest.mark.skipif(_C is None, reason="the CUDA extension is not built")

SIZES = [(600, 512, 50257), (130, 64, 151936), (300, 520, 2500), (129, 128, 16384), (256, 256, 4096), (1, 8, 520),
         (128, 1024, 151936), (8192, 1024, 3072)]


@pytest.mark.parametrize("M,N,K", SIZES)
def test_transposed_a_with_row_major_b_is_not_sliced(M, N, K):
    """A [K, M] with B [N, K] exists with bf16 output only: slices of K, which are fp32 products, cannot run it."""
    assert _C.gemm_plan(M, N, K, a_mn=True, b_mn=False)[0] != "slices"
