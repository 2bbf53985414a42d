"""Quadrature values and their cotangent in H (one kernel) against the Daleckii-Krein
formula in float64 torch, from the same eigendecomposition.

Both evaluate G_ij = sum_ab F_ab u_ia u_jb with the same F (one rounded quotient per
entry), so they differ by the rounding of two sums of k products each:
4 (k + 8) 2^-53 sum_ab |F_ab u_ia u_jb| covers the two orders of summation."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _formula(w, S, fw, fmid, scale):
    s1 = S[:, 0, :]
    d = w[:, :, None] - w[:, None, :]
    same = d.abs() <= 1e-13 * torch.clamp(w.abs()[:, :, None], min=1.0)
    F = torch.where(same, fmid, (fw[:, :, None] - fw[:, None, :]) / torch.where(same, torch.ones_like(d), d))
    U = S * s1[:, None, :]
    G = U @ F @ U.transpose(-1, -2) * scale[:, None, None]
    B = U.abs() @ F.abs() @ U.abs().transpose(-1, -2) * scale[:, None, None]
    return scale * (fw * s1 * s1).sum(-1), G, B


@pytest.mark.parametrize("f,fp", [(torch.log, lambda x: 1.0 / x), (lambda x: x, torch.ones_like)])
@pytest.mark.parametrize("k,p", [(1, 3), (2, 1), (5, 4), (31, 2), (32, 3), (33, 2), (48, 130), (65, 2), (141, 2), (150, 2)])
def test_against_the_formula(k, p, f, fp):
    from matfree_gb300.autodiff import quadform_dH
    from matfree_gb300.funm import tridiag_eigh

    g = torch.Generator().manual_seed(k)
    H = torch.diag_embed(3.0 + torch.rand((p, k), generator=g, dtype=torch.float64))
    if k > 1:
        off = 0.9 * torch.rand((p, k - 1), generator=g, dtype=torch.float64)
        off[:, ::7] = 0.0  # decoupled blocks
        H = H + torch.diag_embed(off, 1) + torch.diag_embed(off, -1)
    if k > 4:
        H[:, 3, 3] = H[:, 2, 2]
    H = H.cuda()
    scale = (1.0 + torch.arange(p, dtype=torch.float64)).cuda()
    values, dH = quadform_dH(H, scale, f, fp)
    w, S = tridiag_eigh(H)
    v, G, B = _formula(w, S, f(w), fp(0.5 * (w[:, :, None] + w[:, None, :])), scale)
    tol = 4 * (k + 8) * 2.0 ** -53
    assert ((values - v).abs() <= tol * scale * f(w).abs().amax(-1)).all()
    i = torch.arange(k)
    want, bound = torch.zeros_like(G), torch.zeros_like(G)
    want[:, i, i], bound[:, i, i] = G[:, i, i], B[:, i, i]
    for a, b in ((i[:-1], i[1:]), (i[1:], i[:-1])):
        want[:, a, b] = 0.5 * (G[:, i[:-1], i[1:]] + G[:, i[1:], i[:-1]])
        bound[:, a, b] = B[:, i[:-1], i[1:]]
    assert ((dH - want).abs() <= tol * bound).all()


def test_differentiable_scale_keeps_the_general_path():
    from matfree_gb300.autodiff import quadform_dH

    H = torch.diag_embed(torch.tensor([[2.0, 3.0, 4.0]], dtype=torch.float64)).cuda()
    scale = torch.tensor([2.0], dtype=torch.float64, device="cuda", requires_grad=True)
    values, dH = quadform_dH(H, scale, torch.log, lambda x: 1.0 / x)
    values.sum().backward()
    torch.testing.assert_close(scale.grad, torch.log(H[:, 0, 0]), rtol=1e-14, atol=0.0)
    fixed = quadform_dH(H, scale.detach(), torch.log, lambda x: 1.0 / x)
    torch.testing.assert_close(fixed[0], values.detach(), rtol=1e-14, atol=0.0)
    torch.testing.assert_close(fixed[1], dH.detach(), rtol=1e-13, atol=1e-15)
