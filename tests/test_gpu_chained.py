"""Launches of a solve's loop that start while the kernel before them ends: the same
bits as with every launch behind the whole of the one before (an event between two
launches, as the profiler records them, forces that).  Every kernel sums in a fixed
order, so the comparison is exact; a read before its data was written would show."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(run):
    from matfree_gb300 import _lib

    lib = _lib.lib()
    lib.mfg_profile_enable(1)
    want = run()
    torch.cuda.synchronize()
    lib.mfg_profile_enable(0)
    for _ in range(8):
        got = run()
        for g, w in zip(got, want):
            assert torch.equal(g, w)


def _dense(n, precision, seed):
    import matfree_gb300 as mf

    g = torch.Generator().manual_seed(seed)
    A = torch.randn((n, n), generator=g, dtype=torch.float64) / n ** 0.5
    A = (A @ A.T + torch.eye(n, dtype=torch.float64)).to(torch.float64 if precision == "fp64" else torch.float32)
    return mf.DenseOperator(A.cuda(), precision=precision, shift=0.5)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16", "bf16x3"])
@pytest.mark.parametrize("n,k,p", [(64, 5, 3), (515, 12, 32), (1100, 9, 150), (2100, 8, 300)])
def test_hessenberg_and_adjoint(n, k, p, precision):
    from matfree_gb300._panel import as_panel
    from matfree_gb300.autodiff import _forward_panels, hessenberg_adjoint

    op = _dense(n, precision, n)
    V = torch.randn((p, n), generator=torch.Generator().manual_seed(1)).cuda()
    panel, ld = as_panel(V, n, op.basis_dtype)
    dH = torch.randn((p, k, k), generator=torch.Generator().manual_seed(2), dtype=torch.float64).cuda()

    def run():
        Q, H, R, c = _forward_panels(op, k, panel, ld)
        Lam, dv = hessenberg_adjoint(op, Q, H, R, c, dH)
        return Q[:, :, :n], H, R[:, :n], c, Lam[:, :, :n], dv[:, :n]  # padding holds no data

    _both(run)


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
def test_product_values(precision):
    from matfree_gb300 import _lib
    from matfree_gb300._panel import as_panel, stream_ptr

    n, k, p = 700, 6, 40
    op = _dense(n, precision, 3)
    V = torch.randn((p, n), generator=torch.Generator().manual_seed(4)).cuda()
    panel, ld = as_panel(V, n, op.basis_dtype)
    lib, s = _lib.lib(), op.c_struct()
    nbytes = lib.mfg_bidiag_workspace_bytes(ctypes.byref(s), ctypes.byref(s), k, p, ld)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")

    def run():
        vals = torch.empty(p, dtype=torch.float64, device="cuda")
        _lib.check(lib.mfg_slq_product(ctypes.byref(s), ctypes.byref(s), k, p, ctypes.c_void_p(panel.data_ptr()), ld,
                                       _lib.MFG_FUN_LOG, 0.0, ctypes.c_void_p(vals.data_ptr()), None,
                                       ctypes.c_void_p(ws.data_ptr()), nbytes, stream_ptr()), "mfg_slq_product")
        return (vals,)

    _both(run)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16x3"])
@pytest.mark.parametrize("n,p", [(130, 1), (3000, 1), (3000, 7), (9000, 2)])
def test_cg(n, p, precision):
    from matfree_gb300 import linalg

    if precision != "bf16x3" and n > 3000:
        pytest.skip("the operators of the other types run the same launches at 3000")
    op = _dense(n, precision, n + p)
    b = torch.randn((p, n), generator=torch.Generator().manual_seed(5)).to(op.basis_dtype).cuda()
    _both(lambda: linalg.cg_batched(op, b, tol=1e-5))


def test_inside_a_stream_capture():
    from matfree_gb300 import _lib
    from matfree_gb300._panel import as_panel, stream_ptr

    n, k, p = 515, 8, 32
    op = _dense(n, "bf16x3", 9)
    V = torch.randn((p, n), generator=torch.Generator().manual_seed(1)).cuda()
    panel, ld = as_panel(V, n, torch.float32)
    lib, s = _lib.lib(), op.c_struct()
    nbytes = lib.mfg_slq_ex_workspace_bytes(ctypes.byref(s), k, p, ld, _lib.MFG_SLQ_TWO_SWEEP)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    vals = torch.empty(p, dtype=torch.float64, device="cuda")

    def run():
        _lib.check(lib.mfg_slq_ex(ctypes.byref(s), k, p, ctypes.c_void_p(panel.data_ptr()), ld, _lib.MFG_FUN_LOG, 0.0,
                                  ctypes.c_void_p(vals.data_ptr()), None, None, None, _lib.MFG_SLQ_TWO_SWEEP,
                                  ctypes.c_void_p(ws.data_ptr()), nbytes, stream_ptr()), "mfg_slq_ex")

    run()
    torch.cuda.synchronize()
    want = vals.clone()
    vals.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(vals, want)
