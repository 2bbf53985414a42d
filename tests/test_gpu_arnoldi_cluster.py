"""The one-launch two-sweep Arnoldi step (a cluster per probe) at the edges of its row splits, rings and
cluster sizes, against the float64 oracle."""

import numpy as np
import pytest
import scipy.sparse as sp
import torch

import matfree_gb300 as mf
from matfree_gb300.decomp import run_hessenberg
from oracle import slq

pytestmark = pytest.mark.gpu


# n: fewer rows than a warp takes, a warp's 256 rows and its neighbours, every number of row warps, ragged rows,
# the largest cluster, the last size of this form and the first past it; p: fewer and more probes than clusters
# fit at a time, of every size; k: no full slot, slots that stay in the ring, slots read again, the deepest
@pytest.mark.parametrize("n,k,p", [(33, 20, 2), (255, 30, 5), (257, 64, 3), (600, 40, 310), (1021, 129, 4), (1023, 33, 160),
                                   (2049, 66, 80), (4098, 100, 40), (5003, 70, 9), (8191, 48, 45), (10001, 16, 9), (16385, 24, 17),
                                   (24577, 9, 3), (32768, 11, 3), (32770, 6, 2)])
def test_cluster_step_matches_oracle(n, k, p):
    rng = np.random.default_rng(n)
    off = -rng.uniform(0.2, 1.0, n - 1)
    far = -rng.uniform(0.1, 0.5, n - 7)
    A = sp.diags([far, off, rng.uniform(3.5, 6.0, n), off, far], [-7, -1, 0, 1, 7], format="csr").astype(np.float32)
    A.sort_indices()
    A64 = A.astype(np.float64)
    V = rng.standard_normal((p, n)).astype(np.float32)
    op = mf.CSROperator.from_scipy(A)
    Q, H, R, c = run_hessenberg(op, k, torch.tensor(V, device="cuda"), reortho="full-two-sweep")
    m = min(p, 4)  # the oracle on the first and last probes
    pick = sorted(set(range(m)) | {p - 1})
    _, Ho, ro, co = slq.hessenberg_forward_batched(lambda X: (A64 @ X.T).T, k, V[pick].astype(np.float64))
    Qc, Hc = Q[pick].double().cpu().numpy(), H[pick].cpu().numpy()
    assert np.abs(Qc @ Qc.transpose(0, 2, 1) - np.eye(k)).max() < 1e-5
    np.testing.assert_allclose(Hc, Ho, rtol=0, atol=1e-4 * np.abs(Ho).max())
    rel = np.stack([(A64 @ x.T).T for x in Qc]) - Hc.transpose(0, 2, 1) @ Qc  # A q_i - sum_l H_li q_l
    rel[:, -1] -= R[pick].double().cpu().numpy()
    assert np.abs(rel).max() < 1e-5 * np.abs(Ho).max()
    np.testing.assert_allclose(c[pick].cpu().numpy(), co, rtol=1e-6)
    # every probe: the tridiagonal part alone gives the same quadrature as the full H
    a = mf.funm.slq_values(op, k, torch.tensor(V, device="cuda"), 0, 0.0).cpu().numpy()
    lam, fsq = mf.funm.tridiag_eigh_first(H)
    b = ((1.0 / (c * c)) * (torch.log(lam) * fsq).sum(-1)).cpu().numpy()
    np.testing.assert_allclose(a, b, rtol=1e-6)
