"""Kernels of a chain of launches start while the kernel before them still writes: what that kernel
writes is not read-only for them.  In every kernel that waits for it (chain_wait) and in the device
functions that such a kernel shares its pointers with, no non-coherent load (__ldg) and no
__restrict__ on a pointer through which another kernel's results are read; the operator, which no
kernel of a loop writes, and pure outputs may have it."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matfree_gb300", "csrc")
OPERATOR = {"Ahi", "Alo"}
OUTPUT = {"W", "values", "eigvals", "first_sq", "status", "nu_last_inv"}
# device functions that are given the pointers of a chained kernel
SHARED = {"gemv_rows", "splitk_reduce", "splitk_shift", "h_scalars"}


def _functions(src):
    """(name, parameters, body) of the functions of a source without comments."""
    src = re.sub(r"//[^\n]*", "", src)
    for m in re.finditer(r"(__global__|__device__ __forceinline__) ([^;{}]*?)\{", src, re.S):
        head = m.group(2)
        at = re.search(r"(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*$", head, re.S)
        if not at:
            continue
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield at.group(1), at.group(2), src[m.end():i]


def _chained():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            src = f.read()
        fns = list(_functions(src))
        for name, params, body in fns:
            if "chain_wait()" in body or name in SHARED or any(s + "<" in body for s in SHARED):
                yield os.path.basename(path), name, params, body


def test_the_chained_kernels_are_found():
    names = {name for _, name, _, _ in _chained()}
    assert {"arnoldi_step_kernel", "arnoldi_h_kernel", "arnoldi_h_band_kernel", "gs_cluster_kernel",
            "dense_tcgen05_splitk_kernel", "dense_tcgen05_pair_kernel", "dense_tcgen05_pair_persistent_kernel",
            "dense_gemv_kernel", "dense_gemv1_kernel", "cg_step_small_kernel", "tridiag_dc_kernel",
            "square_kernel"} | SHARED <= names


@pytest.mark.parametrize("where,name,params,body", [pytest.param(*c, id=c[1]) for c in _chained()])
def test_no_read_only_path_to_what_a_chain_writes(where, name, params, body):
    restricted = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert restricted <= OPERATOR | OUTPUT, (where, name)
    assert "__ldg(" not in body and "__ldcg(" not in body, (where, name)
    assert restricted & OPERATOR or "ld_stream16" not in body
