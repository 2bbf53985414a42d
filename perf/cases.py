"""The calls whose speed this repository is measured by, and the ranges that they stand for.

A case is one call as a user's program makes it: a log-determinant of a kernel
matrix built from points, a sparse or a dense float64 log-determinant, a
training step in the kernel's parameters, a log-determinant of A^T A, a
function of a matrix times vectors, a linear solve.  The sizes are those of the repository's own benchmark and
tests (the serving stream's requests: n from 512 to 32768, depths 16 to 96, 32
to 256 probes) and odd ones between them.

A program whose points, probes and parameters are float32 carries what it gets
in float32, the type that the basis and the products have; a float64 program
carries float64.
"""

import math

import numpy as np
import torch

import matfree_gb300 as mf
from matfree_gb300.autodiff import rbf_logdet

S2, ELL, TAU = 1.0, 0.2, 2.0  # the kernel: variance, length scale, nugget (noisy observations)
HEAT = -0.1  # exp(HEAT x), the serving stream's other function
SHIFT = 0.1  # of the Laplacian


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------


def listed():
    return [
        # the smallest request of the serving stream: launches and latency
        {"name": "logdet small", "kind": "logdet", "n": 512, "k": 16, "p": 32, "fun": "log", "precision": "bf16x3"},
        # an ordinary request of odd size with the stream's other function, a heat trace
        {"name": "heat ragged", "kind": "logdet", "n": 3001, "k": 32, "p": 64, "fun": "exp", "precision": "bf16x3"},
        # the same call with the plain float32 operator
        {"name": "logdet f32", "kind": "logdet", "n": 2000, "k": 32, "p": 64, "fun": "log", "precision": "fp32"},
        # the benchmark's log-determinant
        {"name": "logdet 16k", "kind": "logdet", "n": 16384, "k": 64, "p": 256, "fun": "log", "precision": "bf16x3"},
        # a large, deep request with few probes
        {"name": "logdet deep", "kind": "logdet", "n": 23170, "k": 96, "p": 32, "fun": "log", "precision": "bf16x3"},
        # a training step: log-determinant and its gradient in the kernel's parameters
        {"name": "train 8k", "kind": "train", "n": 8192, "k": 48, "p": 128},
        # the same on a small set of odd size
        {"name": "train small", "kind": "train", "n": 1501, "k": 24, "p": 32},
        # log det(A^T A) by bidiagonalisation
        {"name": "product 8k", "kind": "product", "n": 8192, "k": 32, "p": 128},
        # a sparse operator: shifted 5-point Laplacian on a square grid
        {"name": "laplace 1m", "kind": "sparse", "m": 1024, "k": 100, "p": 64},
        # the plain float64 log-determinant of a dense matrix
        {"name": "dense f64", "kind": "dense64", "n": 1000, "k": 30, "p": 100},
        # a function of a kernel matrix times vectors, here its heat kernel
        {"name": "heat vectors", "kind": "funm", "n": 5000, "k": 40, "p": 48},
        # a linear solve with a kernel matrix by conjugate gradients
        {"name": "solve", "kind": "solve", "n": 8192, "p": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["logdet", "logdet", "logdet", "train", "train", "product", "sparse", "dense64", "funm", "solve"])
    if kind == "logdet":
        c = {"kind": kind, "n": _log_int(rng, 512, 32768), "k": rng.choice([16, 32, 64, 96]),
             "p": rng.choice([32, 64, 128, 256]), "fun": rng.choice(["log", "exp"]), "precision": "bf16x3"}
        if c["n"] <= 4096 and rng.random() < 0.25:
            c["precision"] = "fp32"
        while c["n"] ** 2 * c["k"] * c["p"] > 4e12 and c["p"] > 32:  # no more work than the largest listed one
            c["p"] //= 2
        return c
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 700, 8192), "k": rng.randint(12, 48), "p": _log_int(rng, 16, 128)}
    if kind == "product":
        return {"kind": kind, "n": _log_int(rng, 600, 8192), "k": rng.randint(8, 32), "p": _log_int(rng, 16, 128)}
    if kind == "sparse":
        return {"kind": kind, "m": _log_int(rng, 60, 1024), "k": rng.randint(20, 100), "p": _log_int(rng, 8, 64)}
    if kind == "dense64":
        return {"kind": kind, "n": _log_int(rng, 200, 1500), "k": rng.randint(10, 30), "p": _log_int(rng, 16, 100)}
    if kind == "funm":
        return {"kind": kind, "n": _log_int(rng, 600, 8192), "k": rng.randint(16, 48), "p": _log_int(rng, 8, 64)}
    return {"kind": kind, "n": _log_int(rng, 1000, 12000), "p": rng.choice([1, 1, 2, 4, 8])}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2654435761 % (1 << 31))


def _signs(g, p, n, dtype):
    return torch.randint(0, 2, (p, n), generator=g, device="cuda").to(dtype) * 2 - 1


def _grid_csr(m, weight):
    """CSR of the m x m grid's 5-point operator: `weight` on each edge, the sum of a full row's on the diagonal."""
    idx = torch.arange(m * m, device="cuda").view(m, m)
    rows, cols, vals = [idx.reshape(-1)], [idx.reshape(-1)], [torch.full((m * m,), 4.0 * weight, device="cuda")]
    for a, b in ((idx[:, :-1], idx[:, 1:]), (idx[:-1], idx[1:])):
        for r, c in ((a, b), (b, a)):
            rows.append(r.reshape(-1))
            cols.append(c.reshape(-1))
            vals.append(torch.full((r.numel(),), -weight, device="cuda"))
    rows, cols, vals = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    order = torch.argsort(rows * (m * m) + cols)
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = torch.zeros(m * m + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=m * m), 0)
    return ptr.to(torch.int32), cols.to(torch.int32), vals.to(torch.float32)


def _inputs(case, seed):
    """The plain tensors of a case, made from the seed."""
    g, kind = _generator(seed), case["kind"]
    n, p = case.get("n"), case["p"]
    if kind == "product":
        A = torch.randn((n, n), generator=g, device="cuda") * (0.5 / math.sqrt(n))
        return {"A": A, "probes": _signs(g, p, n, torch.float32)}
    if kind == "sparse":
        weight = float(torch.rand(1, generator=g, device="cuda") * 0.2 + 0.9)
        return {"weight": weight}
    if kind == "dense64":
        B = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64)
        A = B @ B.T / n
        A.diagonal().add_(1.0)
        return {"A": A, "probes": _signs(g, p, n, torch.float64)}
    s = {"x": torch.rand((n, 3), generator=g, device="cuda")}
    if kind == "train":
        start = torch.tensor([0.0, math.log(ELL), math.log(TAU)])
        s["theta"] = start + 0.1 * torch.rand(3, generator=g, device="cuda").cpu()
        s["probes"] = _signs(g, p, n, torch.float32)
    elif kind in ("funm", "solve"):
        s["rhs"] = torch.randn((p, n), generator=g, device="cuda")
    return s


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case, key=mf.prng.prng_key(seed))
    kind = case["kind"]
    if kind in ("logdet", "sparse"):
        n = case["n"] if kind == "logdet" else case["m"] ** 2
        f = mf.funm.funm_exp(HEAT) if case.get("fun") == "exp" else mf.funm.dense_funm_sym_eigh(torch.log)
        s["integrand"] = mf.funm.monte_carlo_funm_sym(f, mf.decomp.tridiag_sym(case["k"]))
        s["sampler"] = mf.stochtrace.sampler_signs(torch.ones(n, device="cuda"), num=case["p"])
        if kind == "sparse":
            s["op"] = mf.CSROperator(*_grid_csr(case["m"], s["weight"]), n, shift=SHIFT)
    elif kind == "product":
        s["op"] = mf.DenseOperator(s.pop("A"), precision="bf16x3", shift=2.0)
        s["op"].transpose()  # kept by the operator
        s["integrand"] = mf.funm.monte_carlo_funm_product_logdet(mf.decomp.bidiag(case["k"]))
    elif kind == "dense64":
        s["op"] = mf.DenseOperator(s.pop("A"), precision="fp64")
        s["integrand"] = mf.funm.monte_carlo_funm_sym_logdet(mf.decomp.tridiag_sym(case["k"]))
    elif kind in ("funm", "solve"):
        s["op"] = mf.RBFKernelOperator(s["x"], s2=S2, ell=ELL, tau=TAU)
        if kind == "funm":
            s["apply"] = mf.funm.funm_lanczos_sym(mf.funm.funm_exp(HEAT), mf.decomp.tridiag_sym(case["k"]))
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "logdet":  # every probe's value: their mean is the estimate, their spread its error
        op = mf.RBFKernelOperator(s["x"], s2=S2, ell=ELL, tau=TAU, precision=case["precision"])
        return s["integrand"].batched(op, s["sampler"](s["key"])).to(s["x"].dtype)
    if kind == "sparse":
        return s["integrand"].batched(s["op"], s["sampler"](s["key"])).to(torch.float32)
    if kind == "product":
        return s["integrand"].batched(s["op"], s["probes"]).to(s["probes"].dtype)
    if kind == "dense64":
        return s["integrand"].batched(s["op"], s["probes"])
    if kind == "train":
        theta = s["theta"].clone().requires_grad_(True)
        value = rbf_logdet(s["x"], theta, s["probes"], case["k"])
        value.backward()
        return {"value": value.detach().to(theta.dtype), "grad": theta.grad}
    if kind == "funm":
        return s["apply"].batched(s["op"], s["rhs"])
    return mf.linalg.cg_batched(s["op"], s["rhs"], tol=1e-5)[0]


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------


def work(case):
    """Inputs once, outputs once, and the arithmetic of the algorithm: one operator product per
    Krylov step (2 n^2 p, or two operations an entry of a sparse row) and two Gram-Schmidt passes
    over the basis (8 n p operations for each earlier vector of a step)."""
    kind, k, p = case["kind"], case.get("k", 0), case["p"]
    n = case["m"] ** 2 if kind == "sparse" else case["n"]
    basis = 4.0 * n * p * k * (k + 1)
    if kind == "logdet":
        return {"bytes": 12.0 * n + 4.0 * p, "flops": 2.0 * n * n * p * k + basis}
    if kind == "train":  # the reverse pass: a product a step, and its own sweeps over the basis
        return {"bytes": 12.0 * n + 4.0 * n * p + 16.0, "flops": 2.0 * (2.0 * n * n * p * k + basis) + 4.0 * n * n * p * k}
    if kind == "product":
        return {"bytes": 4.0 * n * n + 4.0 * n * p + 4.0 * p, "flops": 2.0 * (2.0 * n * n * p * k + basis)}
    if kind == "sparse":
        return {"bytes": 44.0 * n + 4.0 * p, "flops": 10.0 * n * p * k + basis}
    if kind == "dense64":
        return {"bytes": 8.0 * n * n + 8.0 * n * p + 8.0 * p, "flops": 2.0 * n * n * p * k + basis}
    if kind == "funm":
        return {"bytes": 4.0 * n * n + 8.0 * n * p, "flops": 2.0 * n * n * p * k + basis + 2.0 * n * p * k}
    # the number of iterations is the problem's: about sqrt(condition) of them
    its = 0.5 * math.sqrt(0.02 * n / TAU) * math.log(2e5)
    return {"bytes": 4.0 * n * n + 8.0 * n * p, "flops": 2.0 * n * n * p * its}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------


def _kernel64(x, s2, ell, tau):
    """The kernel matrix and the squared distances, float64."""
    x = x.double()
    d2 = sum((x[:, None, i] - x[None, :, i]) ** 2 for i in range(x.shape[1]))
    K = s2 * torch.exp(d2 * (-0.5 / (ell * ell)))
    K.diagonal().add_(tau)
    return K, d2


def _philox_signs(seed, p, n):
    """Philox4x32-10 with counter (element // 4, probe, 0, 0): the top bit of word (element % 4) gives the sign."""
    mask = 0xFFFFFFFF
    groups = (n + 3) // 4
    c0 = torch.arange(groups, device="cuda", dtype=torch.int64)[None, :].expand(p, groups)
    c1 = torch.arange(p, device="cuda", dtype=torch.int64)[:, None].expand(p, groups)
    c2 = torch.zeros_like(c0)
    c3 = torch.zeros_like(c0)
    k0, k1 = int(seed) & mask, int(seed) >> 32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        a, b = 0xD2511F53 * c0, 0xCD9E8D57 * c2  # wraps modulo 2^64: the words below are those of the full product
        c0, c1, c2, c3 = ((b >> 32) & mask) ^ c1 ^ k0, b & mask, ((a >> 32) & mask) ^ c3 ^ k1, a & mask
    words = torch.stack([c0, c1, c2, c3], dim=2).reshape(p, 4 * groups)[:, :n]
    return (1 - 2 * (words >> 31)).double()


def _lanczos64(product, V, k):
    """Basis (p, k, n), diagonals (p, k) and off-diagonals (p, k - 1), and lengths of V's rows, with every vector
    orthogonalised twice against all earlier ones."""
    p, n = V.shape
    Q = torch.zeros((p, k, n), dtype=torch.float64, device=V.device)
    d, e = [], []
    length = V.norm(dim=1)
    q = V / length[:, None]
    for j in range(k):
        Q[:, j] = q
        w = product(q)
        B = Q[:, : j + 1]
        for again in range(2):
            h = torch.bmm(B, w[:, :, None])
            if not again:
                d.append(h[:, j, 0])
            w = w - torch.bmm(h.transpose(1, 2), B)[:, 0]
        beta = w.norm(dim=1)
        if j + 1 < k:
            e.append(beta)
            q = w / beta[:, None]
    d = torch.stack(d, dim=1)
    return Q, d, torch.stack(e, dim=1) if e else d[:, :0], length


def _eigh64(d, e):
    T = torch.diag_embed(d) + torch.diag_embed(e, 1) + torch.diag_embed(e, -1)
    w, S = torch.linalg.eigh(T.cpu())
    return w.to(d.device), S.to(d.device)


def _quadrature64(product, probes, k, f, rows=16):
    """|v|^2 e1^T f(T) e1 for each row v of the probes."""
    got = []
    for i in range(0, probes.shape[0], rows):
        _, d, e, length = _lanczos64(product, probes[i : i + rows].double(), k)
        w, S = _eigh64(d, e)
        got.append(length**2 * (f(w) * S[:, 0] ** 2).sum(-1))
    return torch.cat(got)


class _KernelProduct64(torch.autograd.Function):
    """V K(theta) for float64 rows V, differentiable in V and in theta = (log s2, log ell, log tau)."""

    @staticmethod
    def forward(ctx, V, theta, parts):
        ctx.save_for_backward(V)
        ctx.parts = parts
        return V @ parts[0]

    @staticmethod
    def backward(ctx, g):
        (V,) = ctx.saved_tensors
        K, slope, tau = ctx.parts
        back = g @ K
        nugget = tau * (g * V).sum()
        return back, torch.stack([(back * V).sum() - nugget, ((g @ slope) * V).sum(), nugget]), None


def _train64(case, seed, rows=16):
    s = _inputs(case, seed)
    theta = s["theta"].double()
    s2, ell, tau = (float(t) for t in theta.exp())
    K, d2 = _kernel64(s["x"], s2, ell, tau)
    slope = d2.mul_(1.0 / (ell * ell)).mul_(K)  # zero on the diagonal
    parts = (K, slope, tau)
    theta = theta.cuda().requires_grad_(True)
    values, p = [], case["p"]
    for i in range(0, p, rows):
        V = s["probes"][i : i + rows].double()
        length = V.norm(dim=1)
        q = V / length[:, None]
        Q, d, e = [], [], []
        for j in range(case["k"]):
            Q.append(q)
            w = _KernelProduct64.apply(q, theta, parts)
            B = torch.stack(Q, dim=1)
            for again in range(2):
                h = torch.bmm(B, w[:, :, None])
                if not again:
                    d.append(h[:, j, 0])
                w = w - torch.bmm(h.transpose(1, 2), B)[:, 0]
            beta = w.norm(dim=1)
            if j + 1 < case["k"]:
                e.append(beta)
                q = w / beta[:, None]
        d, e = torch.stack(d, dim=1), torch.stack(e, dim=1)
        T = torch.diag_embed(d) + torch.diag_embed(e, 1) + torch.diag_embed(e, -1)
        w, S = torch.linalg.eigh(T.detach().cpu())
        w, S = w.cuda(), S.cuda()
        # d(e1^T log(T) e1) = <S (F o s1 s1^T) S^T, dT>, F the divided differences of log
        gap = w[:, :, None] - w[:, None, :]
        mid = 0.5 * (w[:, :, None] + w[:, None, :])
        near = gap.abs() <= 1e-6 * mid
        F = torch.where(near, 1.0 / mid, (w.log()[:, :, None] - w.log()[:, None, :]) / torch.where(near, torch.ones_like(gap), gap))
        s1 = S[:, 0]
        G = S @ (F * s1[:, :, None] * s1[:, None, :]) @ S.transpose(1, 2)
        (length[:, None, None] ** 2 * G / p * T).sum().backward()
        values.append(length**2 * (w.log() * s1**2).sum(-1))
    return {"value": torch.cat(values).mean(), "grad": theta.grad.cpu()}


def exact(case, seed):
    kind, k, p = case["kind"], case.get("k"), case["p"]
    if kind == "train":
        return _train64(case, seed)
    s = _inputs(case, seed)
    if kind == "logdet":
        K, _ = _kernel64(s["x"], S2, ELL, TAU)
        f = torch.log if case["fun"] == "log" else lambda w: torch.exp(HEAT * w)
        return _quadrature64(lambda q: q @ K, _philox_signs(seed, p, case["n"]), k, f, rows=64)
    if kind == "sparse":
        m = case["m"]
        w = float(np.float32(s["weight"]))
        diagonal = float(np.float32(4.0 * s["weight"])) + float(np.float32(SHIFT))

        def product(q):
            g = q.view(-1, m, m)
            y = diagonal * g
            y[:, 1:] -= w * g[:, :-1]
            y[:, :-1] -= w * g[:, 1:]
            y[:, :, 1:] -= w * g[:, :, :-1]
            y[:, :, :-1] -= w * g[:, :, 1:]
            return y.view(-1, m * m)

        return _quadrature64(product, _philox_signs(seed, p, m * m), k, torch.log, rows=8)
    if kind == "dense64":
        return _quadrature64(lambda q: q @ s["A"].T, s["probes"], k, torch.log)
    if kind == "product":
        # Lanczos on A^T A gives the bidiagonalisation's B^T B
        A = s["A"].double()
        A.diagonal().add_(2.0)
        return _quadrature64(lambda q: (q @ A.T) @ A, s["probes"], k, torch.log)
    K, _ = _kernel64(s["x"], S2, ELL, TAU)
    V = s["rhs"].double()
    if kind == "solve":
        return torch.linalg.solve(K, V.T).T
    Q, d, e, length = _lanczos64(lambda q: q @ K, V, k)
    w, S = _eigh64(d, e)
    coef = length[:, None] * torch.einsum("pij,pj->pi", S, torch.exp(HEAT * w) * S[:, 0])
    return torch.einsum("pk,pkn->pn", coef, Q)
