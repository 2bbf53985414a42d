"""The split-K cluster form of the tensor-core product at its tile edges."""

import numpy as np
import pytest
import torch

import matfree_gb300 as mf

pytestmark = pytest.mark.gpu


# n: below, at and above a 64-wide K slice, a 128-row tile and two of them, one
# slice per K range, ragged rows; p: the smallest, tile edges, several probe tiles
@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
@pytest.mark.parametrize("n,p", [(9, 9), (63, 16), (64, 17), (65, 128), (127, 129), (129, 31), (257, 300), (511, 32),
                                 (512, 33), (1000, 64), (1025, 9), (2047, 130), (4099, 48), (5120, 256), (9001, 20)])
def test_splitk_product_edges(n, p, precision):
    rng = np.random.default_rng(n + p)
    A = (rng.standard_normal((n, n)) / np.sqrt(n)).astype(np.float32)
    V = rng.standard_normal((p, n)).astype(np.float32)
    shift = 0.75
    op = mf.DenseOperator(torch.tensor(A, device="cuda"), precision=precision, shift=shift)
    got = op.matmat(torch.tensor(V, device="cuda")).double().cpu().numpy()
    again = op.matmat(torch.tensor(V, device="cuda")).double().cpu().numpy()
    assert np.array_equal(got, again)  # fixed-order sums
    stored = op.dense().cpu().numpy()
    if precision == "bf16":
        Vr = torch.tensor(V).bfloat16().double().numpy()
        lost, mats = 0.0, 1
    else:
        Vr, lost, mats = V.astype(np.float64), 3 * 2.0**-16, 3  # lo * lo and the rounding of each lo left out
    E = stored - shift * np.eye(n)
    want = Vr @ E.T + shift * V
    # fp32 accumulation that truncates, one term of a chain per 16 products, then at most 8 chains and the shift
    steps = mats * ((n + 15) // 16) + 16
    bound = (lost + 2.0**-23 * steps) * (np.abs(Vr) @ np.abs(E).T) + 2.0**-23 * np.abs(want)
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()
