"""Gram-Schmidt twice and the adjoint step as one launch each, at the edges of their row splits,
rings and cluster sizes, against the float64 oracle."""

import numpy as np
import pytest
import scipy.sparse as sp
import torch

import matfree_gb300 as mf
from matfree_gb300.autodiff import hessenberg_adjoint
from matfree_gb300.decomp import run_hessenberg
from oracle import adjoint, slq

pytestmark = pytest.mark.gpu


def _banded(n, rng):
    off = -rng.uniform(0.2, 1.0, n - 1)
    far = -rng.uniform(0.1, 0.5, max(n - 7, 0))
    parts, at = [rng.uniform(3.5, 6.0, n), off, off], [0, -1, 1]
    if n > 7:
        parts, at = parts + [far, far], at + [-7, 7]
    A = sp.diags(parts, at, format="csr").astype(np.float32)
    A.sort_indices()
    return A


def _oracle_adjoint(A, Q, H, r, c, dQ, dH, dr, dc):
    """dv and the adjoint states (k, n) of one probe."""
    states = []

    def vjp(q, lam):
        states.append(lam)
        return A.T @ lam, ()

    dv, _ = adjoint.hessenberg_adjoint(vjp, (), Q=Q.T, H=H, r=r, c=c, dQ=dQ.T, dH=dH, dr=dr, dc=dc)
    return dv, np.stack(states[::-1])


def _dense(A, dtype):
    return mf.DenseOperator(torch.tensor(A.toarray(), dtype=dtype, device="cuda"),
                            precision="fp64" if dtype == torch.float64 else "fp32")


# rows: every number of row warps, ragged ends, several cluster sizes; k: no full slot, slots that stay,
# slots read again, more vectors than this form takes; p: fewer and more probes than clusters fit
@pytest.mark.parametrize("dtype,n,k,p", [(torch.float64, 9, 9, 2), (torch.float64, 250, 30, 5), (torch.float64, 515, 64, 3),
                                         (torch.float64, 1030, 40, 310), (torch.float64, 2050, 90, 3),
                                         (torch.float64, 300, 270, 2), (torch.float32, 33, 20, 3),
                                         (torch.float32, 1021, 135, 4), (torch.float32, 2049, 60, 160)])
def test_three_read_form_matches_oracle(dtype, n, k, p):
    rng = np.random.default_rng(n + k)
    A = _banded(n, rng)
    A64 = A.astype(np.float64)
    V = rng.standard_normal((p, n)).astype(np.float32)
    Q, H, R, _ = run_hessenberg(_dense(A, dtype), k, torch.tensor(V, dtype=dtype, device="cuda"), reortho="full")
    pick = sorted({0, 1, p - 1})
    Qc, Hc = Q[pick].double().cpu().numpy(), H[pick].cpu().numpy()
    eps = 1e-13 if dtype == torch.float64 else 1e-5
    assert np.abs(Qc @ Qc.transpose(0, 2, 1) - np.eye(k)).max() < eps * 10
    rel = np.stack([(A64 @ x.T).T for x in Qc]) - Hc.transpose(0, 2, 1) @ Qc
    rel[:, -1] -= R[pick].double().cpu().numpy()
    assert np.abs(rel).max() < 10 * eps * np.abs(Hc).max()
    m = min(k, 60)  # the oracle's H while rounding differences are small
    _, Ho, _, _ = slq.hessenberg_forward_batched(lambda X: (A64 @ X.T).T, m, V[pick].astype(np.float64))
    tol = 1e-9 if dtype == torch.float64 else 1e-3
    np.testing.assert_allclose(Hc[:, :m, :m], Ho, rtol=0, atol=tol * np.abs(Ho).max())


@pytest.mark.parametrize("dtype,n,k,p", [(torch.float64, 12, 6, 2), (torch.float64, 260, 20, 3), (torch.float64, 1100, 33, 2),
                                         (torch.float32, 40, 9, 5), (torch.float32, 600, 40, 160), (torch.float32, 1026, 25, 4),
                                         (torch.float32, 4100, 70, 40), (torch.float32, 9000, 12, 2)])
@pytest.mark.parametrize("with_q", [False, True])
def test_adjoint_step_matches_oracle(dtype, n, k, p, with_q):
    rng = np.random.default_rng(n + k + with_q)
    A = _banded(n, rng)
    A64 = A.astype(np.float64)
    op = _dense(A, dtype) if n <= 2000 else mf.CSROperator.from_scipy(A)
    V = rng.standard_normal((p, n))
    pick = sorted({0, p - 1})
    Qo, Ho, ro, co = slq.hessenberg_forward_batched(lambda X: (A64 @ X.T).T, k, V)
    dH = rng.standard_normal((p, k, k)) / k
    dr = rng.standard_normal((p, n)) / n
    dc = rng.standard_normal(p)
    dQ = rng.standard_normal((p, k, n)) / n if with_q else np.zeros((p, k, n))
    ld = (n + 7) // 8 * 8

    def pad(x):
        out = torch.zeros((*x.shape[:-1], ld), dtype=dtype, device="cuda")
        out[..., :n] = torch.tensor(x, dtype=dtype)
        return out

    t64 = lambda x: torch.tensor(x, dtype=torch.float64, device="cuda")  # noqa: E731
    Lam, dv = hessenberg_adjoint(op, pad(Qo), t64(Ho), pad(ro), t64(co), t64(dH), dr=pad(dr), dc=t64(dc),
                                 dQ=pad(dQ) if with_q else None)
    for b in pick:
        dvo, Lo = _oracle_adjoint(A64, Qo[b], Ho[b], ro[b], co[b], dQ[b], dH[b], dr[b], dc[b])
        tol = 1e-9 if dtype == torch.float64 else 5e-3
        np.testing.assert_allclose(Lam[b, :, :n].double().cpu().numpy(), Lo, rtol=0, atol=tol * np.abs(Lo).max())
        np.testing.assert_allclose(dv[b, :n].double().cpu().numpy(), dvo, rtol=0, atol=tol * np.abs(dvo).max())
