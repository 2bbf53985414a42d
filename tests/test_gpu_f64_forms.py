"""Float64 products at sizes on both sides of the rule between MMAs and FMA tiles, and at the edges of
their tiles, against float64 torch.

Both sum at most n rounded products in some order, the reference too: the results differ by at most
2 (n + 8) 2^-53 of the sum of absolute values."""

import pytest
import torch

import matfree_gb300 as mf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p", [(1, 512), (15, 4200), (31, 1200), (300, 400), (303, 397), (500, 512), (501, 509), (512, 512),
                                 (850, 160), (1000, 100), (1000, 128), (997, 127), (1200, 129), (2000, 64), (2000, 48)])
def test_against_torch(n, p):
    g = torch.Generator(device="cuda").manual_seed(n + p)
    A = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64)
    V = torch.randn((p, n), generator=g, device="cuda", dtype=torch.float64)
    got = mf.DenseOperator(A, precision="fp64", shift=0.25).matmat(V)
    want = V @ A.T + 0.25 * V
    bound = 2 * (n + 8) * 2.0 ** -53 * (V.abs() @ A.abs().T + 0.25 * V.abs())
    assert ((got - want).abs() <= bound).all()
