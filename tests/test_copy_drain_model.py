"""CPU model of the end of a CTA that fills a ring of shared-memory slots by asynchronous copies (the
split-K product and the two cluster kernels): a role that copies, a role that consumes and may give
up at any time, copies that land late.  No copy is in flight when the CTA leaves.

Whether to wait for copies in flight is asked once every role is done.  Asked by the copying role
when it is done itself, it misses a failure of the other role after that."""

import os
import random

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matfree_gb300", "csrc")


def simulate(seed, slots, total, drain):
    """Copies in flight when the CTA leaves.  drain: 'after all roles' or 'in the copying role'."""
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
        if drain == "in the copying role" and failed[0]:
            yield from last_copies(issued)
        count.append(issued)

    def last_copies(issued):
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

    count = []
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
            if not roles and drain == "after all roles" and failed[0]:
                drain = "done"
                roles.append(last_copies(count[0]))
    return len(flying)


@pytest.mark.parametrize("slots,total", [(1, 1), (2, 2), (3, 2), (3, 7), (12, 9), (12, 40)])
def test_no_copy_outlives_the_cta(slots, total):
    assert all(simulate(seed, slots, total, "after all roles") == 0 for seed in range(200))


def test_asking_in_the_copying_role_is_not_enough():
    assert any(simulate(seed, 3, 2, "in the copying role") > 0 for seed in range(200))


@pytest.mark.parametrize("source,kernel", [("arnoldi_cluster.cu", "arnoldi_step_kernel(const"),
                                           ("gs_cluster.cu", "gs_cluster_kernel(const"),
                                           ("dense_tcgen05.cu", "dense_tcgen05_splitk_kernel(const")])
def test_the_kernels_ask_after_their_roles_have_met(source, kernel):
    with open(os.path.join(CSRC, source)) as f:
        body = f.read().split(kernel, 1)[1].split("\n}\n", 1)[0]
    asked = max(body.rfind("(*fail"), body.rfind("&& *abort_flag)"))
    met = max(body.rfind("c_done(S);", 0, asked), body.rfind("cluster_sync_relaxed();", 0, asked))
    drained = body.find("full[", asked)
    assert 0 < met < asked < drained
    assert "full[" not in "".join(x.split(")")[0] for x in body[:met].split("mbar_wait_bounded(")[1:])


def test_every_role_meets():
    for source, kernel in (("arnoldi_cluster.cu", "arnoldi_step_kernel(const"), ("gs_cluster.cu", "gs_cluster_kernel(const")):
        with open(os.path.join(CSRC, source)) as f:
            copy, compute = f.read().split(kernel, 1)[1].split("\n}\n", 1)[0].split("\n  } else {\n    const int wr", 1)
        assert copy.count("c_done(S);") == 1 and compute.count("c_done(S);") == 1
