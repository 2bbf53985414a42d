"""Eigenvalues of the divide and conquer at the rounding of its levels, against Sturm bisection in
numpy's longdouble.

An eigenvalue is rounded once a level, as the sum of a pole and an offset: at most 2^-54 of the
spectral radius each time, 2^-54 / sqrt(3) in the mean, and independently, so the root mean square over
many eigenvalues is about sqrt(levels) 2^-54 / sqrt(3).  Twice that is allowed for the offsets' own
errors.  (A root taken as found while its residual is within k roundings of its terms, but not yet
at their level, is 2 to 4 times as far off.)"""

import math

import numpy as np
import pytest
import torch

from matfree_gb300.funm import tridiag_eigh, tridiag_eigh_first

pytestmark = pytest.mark.gpu


def _below(d, e2, x):
    """Eigenvalues below x (problems, eigenvalues): negative pivots of T - x."""
    q = d[:, 0, None] - x
    count = (q < 0).astype(int)
    for i in range(1, d.shape[1]):
        q = np.where(q == 0, np.longdouble(1e-4000) if np.finfo(np.longdouble).minexp < -10000 else 1e-300, q)
        q = d[:, i, None] - x - e2[:, i - 1, None] / q
        count += q < 0
    return count


def _eigenvalues(d, e):
    """To longdouble's last bits: bisection from the bounds of Gershgorin."""
    d, e = d.astype(np.longdouble), e.astype(np.longdouble)
    k = d.shape[1]
    r = np.abs(d).max(1) + 2 * np.abs(e).max(1)
    lo, hi = np.tile(-r[:, None], (1, k)), np.tile(r[:, None], (1, k))
    want = np.arange(k)[None, :]
    for _ in range(70):
        mid = (lo + hi) / 2
        up = _below(d, e * e, mid) > want
        lo, hi = np.where(up, lo, mid), np.where(up, mid, hi)
    return (lo + hi) / 2


@pytest.mark.parametrize("k", [16, 24, 32])
def test_root_mean_square(k):
    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("longdouble is no longer than double")
    rng = np.random.default_rng(k)
    p = 24
    d, e = rng.standard_normal((p, k)), rng.standard_normal((p, k - 1))
    d[::2], e[::2] = 3.0 + rng.random((p // 2, k)), 0.9 * rng.random((p // 2, k - 1))
    H = torch.as_tensor(d).diag_embed() + torch.as_tensor(e).diag_embed(1) + torch.as_tensor(e).diag_embed(-1)
    want = _eigenvalues(d, e)
    radius = np.abs(want).max(1, keepdims=True)
    bound = 2.0 * math.sqrt(math.ceil(math.log2(k))) * 2.0 ** -54 / math.sqrt(3.0)
    for got in (tridiag_eigh_first(H.cuda())[0], tridiag_eigh(H.cuda())[0]):
        err = ((got.cpu().numpy().astype(np.longdouble) - want) / radius).astype(float)
        assert math.sqrt((err ** 2).mean()) <= bound
