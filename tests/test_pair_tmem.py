"""TMEM of CTA pairs (cta_group::2): allocation, giving up the right to allocate, and release are each
the two CTAs' together.  So both run before either allocates, both hold their columns before either
gives up the right (where no other pair can share the SM), and both have released before either leaves."""

import glob
import os
import random
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matfree_gb300", "csrc")
STEPS = ("tcgen05.alloc.cta_group::2", "tcgen05.relinquish_alloc_permit.cta_group::2", "tcgen05.dealloc.cta_group::2")
MEET = re.compile(r"cluster_sync_(?:all|relaxed)\(\);")


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield re.sub(r"//[^\n]*", "", f.read())


def _body(src, name):
    return src.split(f"{name}(", 1)[1].split("\n}\n", 1)[0]


def test_the_pair_meets_around_each_step_on_its_tmem():
    src = next(s for s in _sources() if "void pair_alloc(" in s)
    alloc, release = _body(src, "void pair_alloc"), _body(src, "void pair_release")
    # meeting, allocation, meeting, right given up (at once where two pairs may share the SM)
    before, rest = alloc.split(STEPS[0])
    shared, rest = rest.split("if (!alone) pair_give_up_right();")
    between, after = rest.split("if (warp == 1 && alone) pair_give_up_right();")
    assert len(MEET.findall(before)) == 1 and len(MEET.findall(between)) == 1
    assert not MEET.search(shared) and not MEET.search(after)
    # meeting, release, meeting
    before, after = release.split(STEPS[2])
    assert len(MEET.findall(before)) == 1 and len(MEET.findall(after)) == 1


def test_every_pair_kernel_goes_through_them():
    text = "".join(_sources())
    assert all(text.count(step) == 1 for step in STEPS)
    kernels = [k.split("\n}\n", 1)[0] for k in text.split("__global__")[1:]]
    pairs = [k for k in kernels if "umma_bf16_pair(" in k]
    assert len(pairs) == 2
    for k in pairs:
        assert k.count("pair_alloc(") == 1 and k.count("pair_release(") == 1
        assert k.rstrip().endswith("warp);") and "return;" not in k
        # the columns released are the ones allocated
        assert re.search(r"pair_alloc\(&sh->tmem_base, ([^;]*), \(uint32_t\)stages \* stage_bytes, warp\);", k).group(1) == re.search(
            r"pair_release\(tmem, ([^;]*), warp\);", k
        ).group(1)


def _run(seed, meetings):
    """Two CTAs take the steps start, allocate, give up, release, leave in any order that the meetings
    (step before which both must have done the one before) allow.  The set of the orders gone wrong."""
    rng, at, bad = random.Random(seed), [0, 0], set()
    while at != [5, 5]:
        c = rng.randrange(2)
        step = at[c] + 1
        if step > 5 or (step in meetings and at[1 - c] < at[c]):
            continue
        if step == 2 and at[1 - c] < 1:
            bad.add("allocates before the peer runs")
        if step == 3 and at[1 - c] < 2:
            bad.add("gives up the right before the peer holds its columns")
        if step == 5 and at[1 - c] < 4:
            bad.add("leaves before the peer has released")
        at[c] = step
    return bad


@pytest.mark.parametrize("left_out", [2, 3, 5])
def test_each_meeting_rules_its_order_out(left_out):
    assert not any(_run(seed, {2, 3, 4, 5}) for seed in range(200))
    assert any(_run(seed, {2, 3, 4, 5} - {left_out}) for seed in range(200))


def test_a_pair_taken_to_be_alone_is_alone():
    least = int(re.search(r"kPairAlone = (\d+) \* 1024", "".join(_sources())).group(1))
    assert 2 * (least + 1) > 228  # a ring of that size and what lies beside it, twice
    for split in (1, 2):
        for bn in range(64, 257, 32):
            stage = split * (128 + bn // 2) * 64
            ring = min(200 * 1024 // stage, 8) * stage
            assert (ring >= least * 1024) == (split == 2 or bn >= 224)


@pytest.mark.gpu
@pytest.mark.parametrize("bn", [64, 96, 128, 160, 192, 224, 0])
@pytest.mark.parametrize("form", [1, 2, 3])
def test_plain_products_of_more_pairs_than_fit(bn, form):
    import matfree_gb300 as mf
    from matfree_gb300 import _lib

    n, p = 5013, 250  # 20 row tiles: up to 160 pairs on 76
    g = torch.Generator(device="cuda").manual_seed(bn + form)
    A = torch.randn((n, n), generator=g, device="cuda")
    V = torch.randn((p, n), generator=g, device="cuda")
    lib = _lib.lib()
    try:
        assert lib.mfg_gemm_tuning_add(n, n, p, p, bn, form) == 0
        got = mf.DenseOperator(A, precision="bf16", shift=0.5).matmat(V).double()
    finally:
        lib.mfg_gemm_tuning_clear()
    a, v = A.bfloat16().double(), V.bfloat16().double()
    want = v @ a.T + 0.5 * V.double()
    # products of bf16 values are exact in float32; each of the n terms is added with one rounding or cut
    bound = n * 2.0 ** -23 * (v.abs() @ a.abs().T) + 2.0 ** -23 * V.double().abs()
    assert ((got - want).abs() <= bound).all()
