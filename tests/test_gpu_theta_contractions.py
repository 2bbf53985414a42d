"""The parameter contractions of the reverse pass on the device: <Lam, A Q>, <Lam, dA Q>
and shift <Lam, Q> against float64 sums of the same products.

Products of floats are summed as two-float pairs: an error of N 2^-48 of sum |lam y| for
the N additions of a thread (at most 64 at these sizes), and the float64 sums above it;
2^-42 sum |lam y| covers both."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(n, p, k, precision, seed, scale=1.0):
    import matfree_gb300 as mf
    from matfree_gb300._panel import padded_ld

    g = torch.Generator().manual_seed(seed)
    x = torch.rand((n, 2), generator=g).cuda()
    op = mf.RBFKernelOperator(x, tau=0.25, precision=precision)
    ld = padded_ld(n)
    Q = torch.randn((p, k, ld), generator=g, dtype=op.basis_dtype).cuda()
    Lam = (scale * torch.randn((p, k, ld), generator=g, dtype=torch.float64)).to(op.basis_dtype).cuda()
    Q[:, :, n:] = 0.0
    Lam[:, :, n:] = float("nan")  # padding is not read as data
    return op, x, Q, Lam


def _want(op, x, Q, Lam):
    from matfree_gb300.autodiff import _rbf_dlogell_operator
    from matfree_gb300.operators import DenseOperator

    n = op.n
    rows = Q.reshape(-1, Q.shape[2])[:, :n]
    lam = Lam.reshape(-1, Q.shape[2])[:, :n].double()
    base = DenseOperator._from_storage(n, op.precision, op.a, op.a_lo, 0.0)
    ys = [base.matmat(rows).double(), _rbf_dlogell_operator(op, x).matmat(rows).double(), op.tau * rows.double()]
    return [((lam * y).sum().item(), (lam * y).abs().sum().item()) for y in ys]


@pytest.mark.parametrize("precision", ["fp32", "bf16", "bf16x3", "fp64"])
@pytest.mark.parametrize("n,p,k", [(1, 1, 1), (5, 1, 3), (1023, 3, 2), (1025, 2, 7), (2052, 40, 4)])
def test_against_float64_sums(n, p, k, precision):
    from matfree_gb300.autodiff import rbf_theta_contractions

    op, x, Q, Lam = _case(n, p, k, precision, 7 * n + k)
    got = rbf_theta_contractions(op, x, Q, Lam).tolist()
    for g, (w, a) in zip(got, _want(op, x, Q, Lam)):
        assert abs(g - w) <= 2.0 ** -42 * a, (g, w, a)


@pytest.mark.parametrize("scale", [1e-36, 1e-28, 1e30, 0.0])
def test_products_outside_the_float_range(scale):
    from matfree_gb300.autodiff import rbf_theta_contractions

    op, x, Q, Lam = _case(300, 4, 3, "fp32", 5, scale)
    got = rbf_theta_contractions(op, x, Q, Lam).tolist()
    for g, (w, a) in zip(got, _want(op, x, Q, Lam)):
        assert abs(g - w) <= 2.0 ** -42 * a, (g, w, a)


def test_mixed_types_and_live_panels_keep_the_general_path():
    from matfree_gb300.autodiff import rbf_theta_contractions

    op, x, Q, Lam = _case(300, 2, 3, "fp32", 6)
    Lam[:, :, 300:] = 0.0
    want = rbf_theta_contractions(op, x, Q, Lam)
    torch.testing.assert_close(rbf_theta_contractions(op, x, Q, Lam.double()), want, rtol=1e-11, atol=1e-9)
    live = Lam.clone().requires_grad_(True)
    rbf_theta_contractions(op, x, Q, live)[2].backward()
    torch.testing.assert_close(live.grad, op.tau * Q, rtol=1e-6, atol=0.0)
