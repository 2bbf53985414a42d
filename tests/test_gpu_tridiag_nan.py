"""NaN in a tridiagonal matrix of a batch: that problem's results are NaN and the solve reports it,
the others keep their bits.  (The sorted merges must not lose an element to a NaN: it would leave a
finite number for a problem that has none, and an unset column index.)"""

import pytest
import torch

import matfree_gb300 as mf
from matfree_gb300 import _lib
from matfree_gb300.funm import slq_values, tridiag_eigh, tridiag_eigh_first

pytestmark = pytest.mark.gpu


def _batch(p, k, seed):
    g = torch.Generator().manual_seed(seed)
    H = torch.diag_embed(3.0 + torch.rand((p, k), generator=g, dtype=torch.float64))
    off = torch.rand((p, k - 1), generator=g, dtype=torch.float64) - 0.5  # both signs: merges run negated too
    return (H + torch.diag_embed(off, 1) + torch.diag_embed(off, -1)).cuda()


@pytest.mark.parametrize("k", [16, 17, 33, 48, 64, 65, 100])
@pytest.mark.parametrize("where", ["diagonal", "last", "off", "inf", "all"])
def test_nan_stays_in_its_problem(k, where):
    H = _batch(4, k, k)
    w0, f0 = tridiag_eigh_first(H)
    l0, S0 = tridiag_eigh(H)
    B = H.clone()
    if where == "diagonal":
        B[1, k // 2, k // 2] = float("nan")
    elif where == "last":
        B[1, k - 1, k - 1] = -float("nan")
    elif where == "off":
        B[1, 2, 3] = float("nan")
    elif where == "inf":
        B[1, 4, 4], B[1, 4, 5] = float("inf"), float("inf")  # inf - inf in the torn leaf
    else:
        B[1] = float("nan")
    w, f = tridiag_eigh_first(B)
    lam, S = tridiag_eigh(B)
    keep = [0, 2, 3]
    assert torch.equal(w[keep], w0[keep]) and torch.equal(f[keep], f0[keep])
    assert torch.equal(lam[keep], l0[keep]) and torch.equal(S[keep], S0[keep])
    assert w[1].isnan().all() and f[1].isnan().all()
    if k <= 64:
        assert lam[1].isnan().all()


@pytest.mark.parametrize("k", [16, 40])
def test_a_solve_with_nan_is_reported(k):
    n = 120
    A = torch.eye(n, device="cuda") * 2.0
    A[7, 9] = A[9, 7] = float("nan")
    op = mf.DenseOperator(A, precision="fp32")
    V = torch.randn((3, n), device="cuda")
    with pytest.raises(RuntimeError, match="did not converge"):
        slq_values(op, k, V, _lib.MFG_FUN_LOG, 0.0)


@pytest.mark.parametrize("k", [20, 48])
def test_an_exhausted_krylov_space_is_still_repeated(k):
    """Five distinct eigenvalues: exact zeros leave NaN behind the request to repeat the solve."""
    n = 256
    d = torch.arange(n, device="cuda") % 5 + 1.0
    op = mf.DenseOperator(torch.diag(d), precision="fp32")
    V = torch.where(torch.arange(3 * n, device="cuda").view(3, n) % 3 == 0, 1.0, -1.0)
    got = slq_values(op, k, V, _lib.MFG_FUN_LOG, 0.0)
    want = slq_values(op, k, V, _lib.MFG_FUN_LOG, 0.0, two_sweep=False)
    torch.testing.assert_close(got, want, rtol=0.0, atol=0.0, equal_nan=True)
