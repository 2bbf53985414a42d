"""A solve whose report is read after what follows it has been enqueued, near an invariant subspace:
the repeat takes the three-sweep form at once (the two-sweep form is deterministic and would ask for
it again), two solves in all, and the results are those of the three-sweep form bit for bit."""

import pytest
import torch

import matfree_gb300 as mf
from matfree_gb300 import _lib, autodiff, decomp
from matfree_gb300.autodiff import rbf_logdet

pytestmark = pytest.mark.gpu


@pytest.fixture
def modes(monkeypatch):
    """The reorthogonalisation forms of the solves, in order (3: two-sweep, 1: three-sweep)."""
    seen, lib = [], _lib.lib()
    solve = lib.mfg_hessenberg
    monkeypatch.setattr(lib, "mfg_hessenberg", lambda *a: (seen.append(a[5]), solve(*a))[1])
    return seen


def _signs(p, n):
    return (torch.randint(0, 2, (p, n), generator=torch.Generator().manual_seed(6)) * 2.0 - 1.0).cuda()


@pytest.mark.parametrize("budget", [None, 1])
def test_logdet(modes, monkeypatch, budget):
    n, k, p = 400, 40, 3
    x = torch.rand((n, 3), generator=torch.Generator().manual_seed(4)).cuda()
    theta = torch.tensor([0.0, 2.0, -3.0], requires_grad=True)  # a long length scale: few eigenvalues above the nugget

    def run():
        value = rbf_logdet(x, theta, _signs(p, n), k, precision="fp32", budget_bytes=budget)
        forward = list(modes)
        (g,) = torch.autograd.grad(value, theta)
        return value.detach(), g, forward

    value, grad, forward = run()
    chunks = p if budget else 1
    assert forward == [3, 1] * chunks
    monkeypatch.setattr(autodiff, "two_sweep_applies", lambda op, k: False)
    modes.clear()
    want, wgrad, forward = run()
    assert forward == [1] * chunks
    assert torch.equal(value, want) and torch.equal(grad, wgrad)


def _low_rank(n, dtype=torch.float32):
    U = torch.randn((n, 6), generator=torch.Generator().manual_seed(2), dtype=torch.float64)
    return (U @ U.T / n + 1e-8 * torch.eye(n, dtype=torch.float64)).to(dtype).cuda()


def test_function_times_vectors(modes, monkeypatch):
    n, k, p = 300, 32, 3
    A, V = _low_rank(n), _signs(p, n)
    f = mf.funm.funm_lanczos_sym(mf.funm.funm_exp(-0.5), mf.decomp.tridiag_sym(k))
    got = f.batched(mf.DenseOperator(A, precision="fp32"), V)
    assert modes == [3, 1]
    monkeypatch.setattr(decomp, "full_reortho", lambda op, k: "full")
    want = f.batched(mf.DenseOperator(A, precision="fp32"), V)
    assert modes == [3, 1, 1]
    assert torch.equal(got, want)


def test_a_callers_matvec_runs_for_two_solves(modes):
    n, k, p = 300, 32, 2
    A, calls = _low_rank(n), []
    op = mf.CallbackOperator(lambda V: (calls.append(1), V @ A)[1], n, batched=True)
    f = mf.funm.funm_lanczos_sym(mf.funm.funm_exp(-0.5), mf.decomp.tridiag_sym(k))
    f.batched(op, _signs(p, n))
    assert modes == [3, 1] and len(calls) == 2 * k
