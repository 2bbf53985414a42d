"""The serving loop never waits for the device: a solve's status word is copied behind it on its
stream and read once its event has completed.  The blocking query inside the loop kept the stall
limit from being looked at when the device did not answer."""

import ctypes

import pytest
import torch

from matfree_gb300 import _lib, serve


class _Event:
    def __init__(self, after):
        self.after = after

    def query(self):
        self.after -= 1
        return self.after < 0


class _Slot:
    busy = False


def _server(monkeypatch, words, after):
    """A server whose solves are events: `words[i]` is the status of launch i, ready after `after[i]` queries."""
    srv = serve.SLQServer.__new__(serve.SLQServer)
    srv.slots, srv.used, srv.budget, srv.precision = [_Slot()], 0.0, 1e12, "bf16x3"
    srv.group_max_n = srv.group_probes = srv.group_members = 0
    launches = []

    def launch(slot, req, flags=None):
        i = len(launches)
        flags = _lib.MFG_SLQ_TWO_SWEEP if flags is None else flags
        launches.append(flags)
        return {"done": _Event(after[i]), "out": torch.tensor([float(i), 0.5]), "flags": flags,
                "word": torch.tensor([words[i]], dtype=torch.int32)}

    class NoWait:
        def __getattr__(self, name):
            assert "status" not in name, "the loop asked the device"
            return getattr(_lib.lib(), name)

    lib = NoWait()
    monkeypatch.setattr(serve._lib, "lib", lambda: lib)
    monkeypatch.setattr(serve, "footprint_bytes", lambda *a: 1.0)
    srv._launch = launch
    return srv, launches


def _request(rid):
    return serve.Request(rid=rid, x=torch.zeros((64, 3)).numpy(), k=8, p=4, fun="log", key=(1, 0))


def test_a_solve_that_asks_for_it_is_repeated_without_a_wait(monkeypatch):
    srv, launches = _server(monkeypatch, [_lib.MFG_ERR_RETRY, _lib.MFG_OK, _lib.MFG_OK], [2, 1, 0])
    res, stats = srv.run([_request(0), _request(1)], realtime=False)
    assert launches == [_lib.MFG_SLQ_TWO_SWEEP, 0, _lib.MFG_SLQ_TWO_SWEEP]
    assert [r.mean for r in res] == [1.0, 2.0] and stats["solves"] == 2


def test_a_stalled_solve_is_reported(monkeypatch):
    srv, _ = _server(monkeypatch, [_lib.MFG_ERR_RETRY], [10 ** 9])
    with pytest.raises(RuntimeError, match="no solve completed"):
        srv.run([_request(0)], realtime=False, stall_s=0.05)


@pytest.mark.gpu
def test_the_copied_word_is_the_status(monkeypatch):
    import matfree_gb300 as mf
    from matfree_gb300._panel import Workspace
    from matfree_gb300.funm import slq_values

    n = 200
    U = torch.randn((n, 10), generator=torch.Generator().manual_seed(0), dtype=torch.float64)
    low_rank = (U @ U.T + 1e-8 * torch.eye(n, dtype=torch.float64)).float().cuda()
    V = torch.randn((2, n), generator=torch.Generator().manual_seed(1)).cuda()
    for A, want in ((low_rank, _lib.MFG_ERR_RETRY), (torch.eye(n, device="cuda") * 2 + low_rank, _lib.MFG_OK)):
        k = 30 if want else 4
        ws = Workspace()
        slq_values(mf.DenseOperator(A, precision="fp32"), k, V, _lib.MFG_FUN_EXP, -1e-3, workspace=ws, two_sweep=True,
                   check=False)
        ptr = ctypes.c_void_p(ws.buf.data_ptr())
        word = serve._status_word(ptr, torch.cuda.current_stream())
        torch.cuda.synchronize()
        assert int(word[0]) == want == _lib.lib().mfg_workspace_status(ptr, None)
