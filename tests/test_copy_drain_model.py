"""CPU model of the end of a CTA that fills a ring of shared-memory slots by asynchronous copies (the
split-K product and the two cluster kernels): a role that copies, a role that consumes and may give
up at any time, copies that land late.  No copy is in flight when the CTA leaves.

The copying role waits for its last fills whatever has happened so far.  A wait that depends on a
failure seen by then is not enough: the other role may give up after it."""

import os
import random

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matfree_gb300", "csrc")


def simulate(seed, slots, total, drain):
    """Copies in flight when both roles are done.  drain: 'always' or 'if failed'."""
    rng = random.Random(seed)
    landed, freed, failed = set(), set(), [False]
    flying = []
    gives_up = rng.choice([None, rng.randrange(total)])  # the consumer's last slice

    def copier():
        issued = 0
        for f in range(total):
            while f >= slots and f - slots not in freed:
                if failed[0]:
                    break
                yield
            else:
                flying.append(f)
                issued += 1
                yield
                continue
            break
        if drain == "always" or failed[0]:
            for f in range(max(0, issued - slots), issued):
                while f not in landed:
                    yield

    def consumer():
        for f in range(total):
            while f not in landed:
                if f == gives_up and rng.random() < 0.3:  # its wait ran out
                    failed[0] = True
                    return
                yield
            if f == gives_up:
                failed[0] = True
                return
            freed.add(f)
            yield

    roles = [copier(), consumer()]
    while roles:
        if flying and rng.random() < 0.25:
            landed.add(flying.pop(rng.randrange(len(flying))))
            continue
        role = rng.choice(roles)
        try:
            next(role)
        except StopIteration:
            roles.remove(role)
    return len(flying)


@pytest.mark.parametrize("slots,total", [(1, 1), (2, 2), (3, 2), (3, 7), (12, 9), (12, 40)])
def test_no_copy_outlives_the_cta(slots, total):
    assert all(simulate(seed, slots, total, "always") == 0 for seed in range(200))


def test_a_wait_for_failures_seen_so_far_is_not_enough():
    assert any(simulate(seed, 3, 2, "if failed") > 0 for seed in range(200))


@pytest.mark.parametrize("source,kernel", [("arnoldi_cluster.cu", "arnoldi_step_kernel(const"),
                                           ("gs_cluster.cu", "gs_cluster_kernel(const"),
                                           ("dense_tcgen05.cu", "dense_tcgen05_splitk_kernel(const")])
def test_the_kernels_wait_for_their_copies_in_any_case(source, kernel):
    with open(os.path.join(CSRC, source)) as f:
        body = f.read().split(kernel, 1)[1].split("__global__", 1)[0]
    assert "mbar_wait_bounded(" in body
    assert "if (*fail" not in body and "if (*abort_flag" not in body
