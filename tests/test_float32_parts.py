"""The sum of three bfloat16 numbers that a float32 number is split into for the tensor cores: what the split keeps, and that the
tests' bound on a product's error (``NORM`` in test_gpu_float32_kernels.py) would notice any one of its six terms missing."""
import pytest
import torch

from test_gpu_float32_kernels import NORM, SHAPES, TERMS, operands, split_in_three


@pytest.mark.parametrize("M, N, K", SHAPES)
def test_every_term_of_the_product_counts(M, N, K):
    a, w = operands(M, N, K)
    pa, pw = split_in_three(a), split_in_three(w)
    want = a.double() @ w.double().t()
    terms = {(i, j): pa[i] @ pw[j].t() for i, j in TERMS}
    error = lambda sums: float((sums - want).norm() / want.norm())
    assert error(sum(terms.values())) < 0.1 * NORM
    for missing in TERMS:
        assert error(sum(t for k, t in terms.items() if k != missing)) > 2 * NORM


def test_the_split_loses_nothing():
    g = torch.Generator().manual_seed(1)
    for exponent in (-149, -140, -126, -112, -60, 0, 60, 102):
        x = (torch.rand(1000, generator=g) + 1) * torch.tensor(2.0 ** exponent, dtype=torch.float64).float()
        assert torch.equal(sum(split_in_three(x)), x.double())
