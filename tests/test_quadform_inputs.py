"""What the quadrature's cotangent and the hyper-parameter contractions take from their callers:
f, f' and scale of any shape, type and device that the torch operations of the general path take,
followed by gradients, forward-mode tangents or a function transform or not.

The kernel reads whole (p, k), (p, k, k) and (p,) float64 arrays, so only those may reach it.
Against the general path, run here by a scale that asks for a gradient: the same operations, whose
sums may be taken in another order, at most 4 (k + 8) 2^-53 k max |F| for orthonormal S and scale 1."""

import pytest
import torch
import torch.autograd.forward_ad as fwad

from matfree_gb300.autodiff import _plain, _plain_float64


def test_plain_tensors():
    t, cpu = torch.ones(3, dtype=torch.float64), torch.device("cpu")
    assert _plain_float64(cpu, t, t.clone())
    assert not _plain_float64(cpu, t, 1.0)
    assert not _plain_float64(cpu, t.float())
    assert not _plain_float64(torch.device("cuda", 0), t)
    live = t.clone().requires_grad_()
    assert not _plain(live)
    with torch.no_grad():
        assert _plain(live)
    with fwad.dual_level():
        assert not _plain(fwad.make_dual(t, t))
    assert _plain(t)
    seen = []
    torch.vmap(lambda x: (seen.append(_plain(x)), x)[1])(t)
    torch.func.jvp(lambda x: (seen.append(_plain(x)), x)[1], (t,), (t,))
    assert seen == [False, False]


def _problem(p=5, k=24):
    g = torch.Generator().manual_seed(7)
    H = torch.diag_embed(3.0 + torch.rand((p, k), generator=g, dtype=torch.float64))
    off = 0.9 * torch.rand((p, k - 1), generator=g, dtype=torch.float64)
    H = H + torch.diag_embed(off, 1) + torch.diag_embed(off, -1)
    return H.cuda(), torch.ones(p, dtype=torch.float64, device="cuda")


def _general(H, scale, f, fp):
    from matfree_gb300.autodiff import quadform_dH

    values, dH = quadform_dH(H, scale.clone().requires_grad_(), f, fp)
    return values.detach(), dH.detach()


@pytest.mark.gpu
@pytest.mark.parametrize("f,fp,peak", [
    (lambda w: w.mean(0, keepdim=True).log(), lambda x: 1.0 / x, 1e3),  # one row for all problems
    (lambda w: torch.full((1, w.shape[1]), 2.0, dtype=w.dtype, device=w.device), torch.zeros_like, 1.0),
    (lambda w: w.sum(1, keepdim=True), lambda x: torch.ones(1, dtype=x.dtype, device=x.device), 1.0),  # one value a problem
    (lambda w: w, lambda x: 1.0, 1.0),  # a number for f'
    (lambda w: w, lambda x: torch.ones((), dtype=x.dtype), 1.0),  # a number on the host
    (lambda w: w.float(), lambda x: torch.ones_like(x), 1.0),
], ids=["row", "constant row", "column", "number", "host number", "float32"])
def test_broadcast_inputs_keep_their_values(f, fp, peak):
    from matfree_gb300.autodiff import quadform_dH

    H, scale = _problem()
    k = H.shape[1]
    (v, dH), (v0, dH0) = quadform_dH(H, scale, f, fp), _general(H, scale, f, fp)
    tol = 4 * (k + 8) * 2.0 ** -53 * k * peak
    torch.testing.assert_close(v, v0, rtol=tol, atol=tol)
    torch.testing.assert_close(dH, dH0, rtol=tol, atol=tol)


@pytest.mark.gpu
def test_values_on_the_host_are_refused():
    from matfree_gb300.autodiff import quadform_dH

    H, scale = _problem()
    for args in ((H, scale, lambda w: w.cpu(), torch.ones_like), (H, scale.cpu(), torch.log, lambda x: 1.0 / x),
                 (H, scale, torch.log, lambda x: (1.0 / x).cpu())):
        with pytest.raises(RuntimeError):
            quadform_dH(*args)


@pytest.mark.gpu
def test_tangents_of_scale_and_parameters_of_the_derivative():
    from matfree_gb300.autodiff import quadform_dH

    H, scale = _problem()
    with fwad.dual_level():
        values, _ = quadform_dH(H, fwad.make_dual(scale, torch.ones_like(scale)), torch.log, lambda x: 1.0 / x)
        v, t = fwad.unpack_dual(values)
        torch.testing.assert_close(t, v, rtol=1e-13, atol=1e-13)  # the values are linear in scale = 1
    live = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
    _, dH = quadform_dH(H, scale, lambda w: w, lambda x: live * torch.ones_like(x))
    assert dH.requires_grad  # a parameter of f' alone


@pytest.mark.gpu
def test_contractions_with_a_sparse_derivative():
    import matfree_gb300 as mf
    from matfree_gb300.autodiff import rbf_theta_contractions

    n, ld = 40, 40
    g = torch.Generator(device="cuda").manual_seed(3)
    op = mf.RBFKernelOperator(torch.rand((n, 3), generator=g, device="cuda"), precision="fp32")
    Q, Lam = (torch.randn((2, 3, ld), generator=g, device="cuda") for _ in range(2))
    i = torch.arange(n + 1, device="cuda", dtype=torch.int32)
    dl = mf.CSROperator(i, i[:-1], torch.full((n,), 2.0, device="cuda"), n)  # 2 I
    got = rbf_theta_contractions(op, op.x, Q, Lam, dl=dl)[1]
    torch.testing.assert_close(got, 2.0 * (Q.double() * Lam.double()).sum(), rtol=1e-6, atol=1e-5)
