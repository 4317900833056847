"""The cluster form's sums (cluster_sum in cgxx_b200/csrc/gridred.cuh) as a small
model, run over random interleavings of the CTAs (no GPU): a CTA's shared memory is
written only while that CTA runs, and no partial is overwritten before it is read.
Whether a kernel meets at a cluster barrier before its first sum and before its end
is taken from its source."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "cgxx_b200", "csrc")
KERNELS = [("solve64.cuh", "k_solve64"), ("persist.cuh", "k_inner_split"),
           ("persist.cuh", "k_inner_fused")]
# A barrier that every cluster launch passes, whatever its matrix.
BARRIER = r"if \((PERM \|\| )?CLUSTER\)\s+(ok = sync_over<CLUSTER|cluster_sync\(\))"


def end_barriers(file, kernel):
    with open(os.path.join(CSRC, file)) as f:
        src = f.read()
    src = src[re.search(r"\b%s\([^;{]*\{" % kernel, src).end():]
    src = re.sub(r"//[^\n]*", "", src[:src.index("\n}\n")])
    enter = re.search(BARRIER, src[:src.index("sum_over<")])
    leave = re.search(BARRIER, src[src.rindex("sum_over<"):])
    return bool(enter), bool(leave)


class Fault(Exception):
    pass


def cta(c, rounds, enter, leave, running, part):
    """One CTA, step by step; True where it waits at the cluster's barrier."""
    running[c] = True
    yield enter
    for r in range(rounds):
        for t in range(len(running)):
            if not running[t]:
                raise Fault(f"CTA {c} stores to CTA {t}, which does not run")
            part[t][r & 1][c] = r
            yield False
        yield True
        if part[c][r & 1] != [r] * len(running):
            raise Fault(f"CTA {c} reads a partial of another round")
        yield False
    yield leave
    running[c] = False


def run(ctas, rounds, enter, leave, rng):
    running = [False] * ctas
    part = [[[None] * ctas, [None] * ctas] for _ in range(ctas)]
    live = {c: cta(c, rounds, enter, leave, running, part) for c in range(ctas)}
    waiting = set()
    while live:
        if waiting == set(live):
            waiting.clear()
        c = rng.choice(sorted(set(live) - waiting))
        try:
            if next(live[c]):
                waiting.add(c)
        except StopIteration:
            del live[c]


@pytest.mark.parametrize("file,kernel", KERNELS)
def test_cluster_sums_write_to_running_ctas_only(file, kernel):
    enter, leave = end_barriers(file, kernel)
    for ctas in (2, 3, 5):
        for seed in range(200):
            run(ctas, 5, enter, leave, random.Random(seed))


def test_the_model_sees_a_missing_barrier():
    with pytest.raises(Fault):
        for seed in range(200):
            run(3, 5, False, True, random.Random(seed))
