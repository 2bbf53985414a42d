"""The divide-and-conquer eigensolver at each number of lanes per root (chosen from k and the
number of problems), with merges that deflate beside merges that do not."""

import numpy as np
import pytest
import torch

import matfree_gb300 as mf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,p", [(16, 3), (16, 400), (17, 160), (31, 310), (33, 2), (45, 153), (64, 305), (65, 7),
                                 (100, 160), (130, 2)])
def test_groups_of_lanes_match_eigh(k, p):
    rng = np.random.default_rng(k * 1000 + p)
    d = rng.uniform(0.5, 4.0, (p, k))
    e = rng.uniform(-1.0, 1.0, (p, k - 1))
    e[1::3, k // 2] = 0.0  # a coupling that is torn for good
    d[2::3, 1:] = d[2::3, :1]  # equal poles in every merge
    e[::5] *= 1e-9  # nearly decoupled
    T = np.zeros((p, k, k))
    i = np.arange(k)
    T[:, i, i] = d
    T[:, i[:-1], i[1:]] = T[:, i[1:], i[:-1]] = e
    w, S = np.linalg.eigh(T)
    lam, fsq = (t.cpu().numpy() for t in mf.funm.tridiag_eigh_first(torch.tensor(T, device="cuda")))
    scale = np.abs(w).max()
    assert np.abs(lam - w).max() <= 1e-12 * scale
    assert np.abs(fsq.sum(-1) - 1.0).max() <= 1e-12
    for g in (np.exp, np.cos, lambda x: x * x):
        got, want = (g(lam) * fsq).sum(-1), (g(w) * S[:, 0] ** 2).sum(-1)
        assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(g(w)).max())
    if k <= 64:
        v, Q = (t.cpu().numpy() for t in mf.funm.tridiag_eigh(torch.tensor(T, device="cuda")))
        assert np.abs(Q.transpose(0, 2, 1) @ Q - np.eye(k)).max() <= 1e-12 * k
        assert np.abs((Q * v[:, None, :]) @ Q.transpose(0, 2, 1) - T).max() <= 1e-12 * k * scale


@pytest.mark.parametrize("k", [16, 33, 64, 100])
@pytest.mark.parametrize("exponent", [-400, 0, 400])
def test_scaled_problems_have_scaled_eigenvalues(k, exponent):
    """The float32 first steps run on poles scaled to 1: powers of two do not change a result beyond the
    tolerances of the equal-scale test.  (Squares of distances leave the float64 range past 2^-500 and 2^500.)"""
    rng = np.random.default_rng(k)
    d = rng.uniform(0.5, 4.0, (6, k))
    e = rng.uniform(-1.0, 1.0, (6, k - 1)) * 10.0 ** rng.integers(-13, 1, (6, k - 1))
    i = np.arange(k)
    T = np.zeros((6, k, k))
    T[:, i, i] = d
    T[:, i[:-1], i[1:]] = T[:, i[1:], i[:-1]] = e
    w, S = np.linalg.eigh(T)
    lam, fsq = (t.cpu().numpy() for t in mf.funm.tridiag_eigh_first(torch.tensor(np.ldexp(T, exponent), device="cuda")))
    lam = np.ldexp(lam, -exponent)
    assert np.abs(lam - w).max() <= 1e-12 * np.abs(w).max()
    got, want = (np.exp(lam) * fsq).sum(-1), (np.exp(w) * S[:, 0] ** 2).sum(-1)
    assert np.abs(got - want).max() <= 1e-12 * np.exp(w).max()
