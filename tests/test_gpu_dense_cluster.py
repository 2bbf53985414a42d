"""The float32 and float64 dense products at the edges of their tiles, slices and K ranges."""

import numpy as np
import pytest
import torch

import matfree_gb300 as mf

pytestmark = pytest.mark.gpu


# n: one slice and less, slice and tile edges, fewer slices than K ranges, ragged rows and columns;
# p: single, tile edges, several tiles
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n,p", [(1, 1), (7, 3), (16, 8), (31, 9), (33, 33), (64, 64), (65, 31), (127, 65), (257, 7),
                                 (300, 256), (700, 37), (1000, 100), (1203, 60), (2050, 16)])
def test_dense_product_edges(n, p, precision):
    rng = np.random.default_rng(n * 7 + p)
    dt = np.float32 if precision == "fp32" else np.float64
    A = rng.standard_normal((n, n)).astype(dt)
    V = rng.standard_normal((p, n)).astype(dt)
    op = mf.DenseOperator(torch.tensor(A, device="cuda"), precision=precision, shift=-0.5)
    got = op.matmat(torch.tensor(V, device="cuda"))
    assert torch.equal(got, op.matmat(torch.tensor(V, device="cuda")))  # fixed-order sums
    A, V = A.astype(np.longdouble), V.astype(np.longdouble)
    want = V @ A.T - np.longdouble(0.5) * V
    # n + 9 roundings of sums no larger than |V| |A|^T
    bound = (n + 9) * np.finfo(dt).eps * (np.abs(V) @ np.abs(A).T + np.abs(V))
    assert (np.abs(got.cpu().numpy().astype(np.longdouble) - want) <= bound).all()


def test_dense_product_ignores_padding_columns():
    # the storage's columns past n are not data, whatever they hold
    n, p = 67, 5
    rng = np.random.default_rng(0)
    for precision, dt in (("fp32", torch.float32), ("fp64", torch.float64)):
        A = torch.tensor(rng.standard_normal((n, n)), dtype=dt, device="cuda")
        V = torch.tensor(rng.standard_normal((p, n)), dtype=dt, device="cuda")
        op = mf.DenseOperator(A, precision=precision)
        want = op.matmat(V)
        op.a[:, n:] = float("nan")
        panel = torch.full((p, 72), float("nan"), dtype=dt, device="cuda")
        panel[:, :n] = V
        assert torch.equal(op.matmat(panel[:, :n]), want)
