"""Plans of the one-launch steps (mfg_step_plan, host arithmetic; no GPU) for tables of the clusters
that a GPU holds: a size that the GPU does not hold is not chosen, and where none is left the answer
is 0, on which the solves take the separate launches instead of refusing the call.  A plan covers
the rows and its shared memory is within what the kernels are allowed."""

import ctypes
import random

import numpy as np
import pytest

from matfree_gb300 import _lib

SIZES = [1, 2, 4, 6, 8, 10, 12, 14, 16]
ALL = [304, 152, 74, 48, 36, 28, 24, 20, 14]  # a GB300's
MAX_ROWS = 2048
PREC = {"float": _lib.MFG_PREC_FP32, "double": _lib.MFG_PREC_FP64}


def plan(kind, prec, n, p, ncols, table):
    t = np.ascontiguousarray(np.broadcast_to(np.asarray(table, dtype=np.int32), (4, 9)))
    out = np.zeros(4, dtype=np.int32)
    S = _lib.lib().mfg_step_plan(kind, PREC[prec], n, p, ncols, ctypes.c_void_p(t.ctypes.data),
                                 ctypes.c_void_p(out.ctypes.data))
    return S, out


def without(*sizes):
    return [0 if s in sizes else c for s, c in zip(SIZES, ALL)]


@pytest.mark.parametrize("kind,prec", [(0, "float"), (1, "float"), (1, "double"), (2, "float"), (2, "double")])
def test_no_cluster_of_16_leaves_the_largest_sizes_to_the_separate_launches(kind, prec):
    for n in (28673, 30000, 32768):
        assert plan(kind, prec, n, 15, 8, ALL)[0] == 16
        assert plan(kind, prec, n, 15, 8, without(16))[0] == 0
    for n in (512, 8192, 28672):
        assert 0 < plan(kind, prec, n, 15, 8, without(16))[0] < 16


@pytest.mark.parametrize("kind,prec", [(0, "float"), (1, "float"), (1, "double"), (2, "float"), (2, "double")])
def test_nothing_held_is_no_plan(kind, prec):
    for n in (1, 512, 32768):
        assert plan(kind, prec, n, 4, 3, [0] * 9)[0] == 0


def test_limits_of_the_kernels():
    assert plan(0, "float", 32769, 8, 4, ALL)[0] == 0
    assert plan(1, "float", 32769, 8, 4, ALL)[0] == 0
    assert plan(0, "float", 1000, 8, 129, ALL)[0] == 0
    assert plan(0, "double", 1000, 8, 4, ALL)[0] == 0  # float bases only
    assert plan(1, "float", 1000, 8, 257, ALL)[0] == 0
    assert plan(2, "float", 1000, 8, 129, ALL)[0] == 0
    assert plan(2, "float", 1000, 8, 128, ALL)[0] > 0


@pytest.mark.parametrize("kind,prec", [(0, "float"), (1, "float"), (1, "double"), (2, "float"), (2, "double")])
def test_a_plan_covers_the_rows_with_a_size_that_is_held(kind, prec):
    rng = random.Random(kind)
    for _ in range(400):
        table = [c if rng.random() < 0.6 else 0 for c in ALL]
        n, p = rng.randint(1, 32768), rng.choice([1, 3, 15, 40, 128, 700])
        ncols = rng.randint(1, 128)
        S, (s, R, warps, slots) = plan(kind, prec, n, p, ncols, table)
        room = [z for z, c in zip(SIZES, table) if c and -(-n // z) <= MAX_ROWS]
        if S == 0:
            if kind == 0:  # its shared memory does not depend on the vectors
                assert not room
            continue
        assert S == s and S in room
        assert S * R >= n and R % 4 == 0 and R <= 256 * warps <= MAX_ROWS
        assert slots >= 1
