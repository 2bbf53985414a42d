"""Products with two to eight vectors around the size from which some forms take one row a warp in
place of two, against float64.

A result is a float32 sum of at most 24 ceil(n / 256) products a lane and 16 more additions, each
rounded by 2^-24 of the sum of absolute values; a split operator and vector leave 2^-16 of each
product apart (two truncated pairs and their lowest product)."""

import math

import pytest
import torch

import matfree_gb300 as mf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(8999, "bf16"), (9000, "bf16"), (9001, "bf16"), (9016, "bf16"),
                                         (10999, "bf16x3"), (11000, "bf16x3"), (11001, "bf16x3"), (11016, "bf16x3")])
def test_around_the_border(n, precision):
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), generator=g, device="cuda")
    op = mf.DenseOperator(A, precision=precision, shift=0.5)
    for p in (2, 3, 4, 5, 6, 8):
        V = torch.randn((p, n), generator=g, device="cuda")
        got = op.matmat(V).double()
        rows = torch.cat([torch.arange(0, n, 997, device="cuda"), torch.arange(n - 9, n, device="cuda")])
        a, v = A[rows], V
        if precision == "bf16":
            a, v = a.bfloat16(), v.bfloat16()
        a, v = a.double(), v.double()
        want = v @ a.T + 0.5 * V[:, rows].double()
        bound = ((24 * math.ceil(n / 256) + 16) * 2.0 ** -24 + (2.0 ** -16 if precision == "bf16x3" else 0.0)) \
            * (v.abs() @ a.abs().T) + 2.0 ** -24 * V[:, rows].abs()
        assert ((got[:, rows] - want).abs() <= bound).all()
