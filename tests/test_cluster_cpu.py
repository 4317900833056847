"""The persistent solves' sums and barriers (cgxx_b200/csrc/gridred.cuh) as small
models, run over random interleavings of the CTAs (no GPU).

cluster_sum: a CTA's shared memory is written only while that CTA runs; whether a
kernel meets at a cluster barrier before its first sum and before its end is taken
from its source. All forms: no partial sum is overwritten before every CTA has read
it, and a CTA reads of the CTAs below what wait_below promises."""
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


# One iteration of each kernel: sums of one or two values, barriers, and the neighbour
# wait (write y, wait_below, read y of the CTAs below).
FORMS = {"fused": [1, 2], "split": [1, 2, "barrier"], "learned fused": [1, "below", 2],
         "learned split": [1, 1, "barrier", 1, "barrier"]}
ITERATIONS = 4


class Cluster:
    """cluster_sum: a set of partials per kind of sum and round parity in every CTA."""

    def __init__(self, ctas, enter=True):
        self.ctas, self.enter = ctas, enter
        self.running = [False] * ctas
        self.part = [{} for _ in range(ctas)]
        self.waiting = set()

    def barrier(self, c):
        self.waiting.add(c)
        if len(self.waiting) == self.ctas:
            self.waiting = set()
        while c in self.waiting:
            yield

    def start(self, c):
        self.running[c] = True
        if self.enter:
            yield from self.barrier(c)

    def sum(self, c, rnd, nv):
        for t in range(self.ctas):
            if not self.running[t]:
                raise Fault(f"CTA {c} stores to CTA {t}, which does not run")
            self.part[t].setdefault((nv, rnd & 1), [None] * self.ctas)[c] = rnd
            yield
        yield from self.barrier(c)
        if self.part[c][nv, rnd & 1] != [rnd] * self.ctas:
            raise Fault(f"CTA {c} reads a partial of another round")
        return rnd + 1

    def sync(self, c, rnd):
        yield from self.barrier(c)
        return rnd

    def below(self, c, it, n):
        yield from self.barrier(c)


class Grid:
    """grid_sum: one counter, two sets of partials by round parity; wait_below: a flag
    per CTA."""

    def __init__(self, ctas):
        self.ctas, self.count, self.flags = ctas, 0, [0] * ctas
        self.part = [[None] * ctas, [None] * ctas]

    def start(self, c):
        yield

    def sum(self, c, rnd, nv):
        if nv:
            self.part[rnd & 1][c] = rnd
        yield
        self.count += 1
        while self.count < (rnd + 1) * self.ctas:
            yield
        for t in range(self.ctas if nv else 0):
            if self.part[rnd & 1][t] != rnd:
                raise Fault(f"CTA {c} reads a partial of another round")
            yield
        return rnd + 1

    def sync(self, c, rnd):
        return (yield from self.sum(c, rnd, 0))

    def below(self, c, it, n):
        self.flags[c] = it + 1
        for b in range(max(0, c - n), c):
            while self.flags[b] < it + 1:
                yield


def cta(mem, c, form, y, n):
    yield from mem.start(c)
    rnd = 0
    for it in range(ITERATIONS):
        for step in FORMS[form]:
            if step == "barrier":
                rnd = yield from mem.sync(c, rnd)
            elif step == "below":
                y[c] = it
                yield
                yield from mem.below(c, it, n)
                for b in range(max(0, c - n), c):
                    if y[b] != it:
                        raise Fault(f"CTA {c} reads y of CTA {b} from another iteration")
                    yield
            else:
                rnd = yield from mem.sum(c, rnd, step)
    if isinstance(mem, Cluster):
        yield from mem.barrier(c)
        mem.running[c] = False


def run(mem, form, seed, n=2):
    rng = random.Random(seed)
    y = [None] * mem.ctas
    live = {c: cta(mem, c, form, y, n) for c in range(mem.ctas)}
    while live:
        c = rng.choice(sorted(live))
        # Some CTAs run on for a while: the far ahead and the left behind.
        for _ in range(rng.choice([1, 1, 5, 40])):
            try:
                next(live[c])
            except StopIteration:
                del live[c]
                break


@pytest.mark.parametrize("file,kernel", KERNELS)
def test_cluster_sums_write_to_running_ctas_only(file, kernel):
    enter, leave = end_barriers(file, kernel)
    assert leave
    forms = {"k_solve64": ("fused", "split"), "k_inner_split": ("split", "learned split"),
             "k_inner_fused": ("fused", "learned fused")}[kernel]
    for form in forms:
        for ctas in (2, 3, 5):
            for seed in range(100):
                run(Cluster(ctas, enter), form, seed)


@pytest.mark.parametrize("form", FORMS)
def test_grid_sums_read_before_reuse(form):
    for ctas in (2, 3, 6):
        for seed in range(100):
            run(Grid(ctas), form, seed)


def test_the_models_see_what_is_missing(monkeypatch):
    def faults(make, form):
        with pytest.raises(Fault):
            for seed in range(200):
                run(make(), form, seed)
    faults(lambda: Cluster(3, enter=False), "fused")
    # One set of partials instead of two.
    one = Grid(3)
    one.part[1] = one.part[0]
    faults(lambda: setattr(one, "count", 0) or one, "learned split")
    # No wait for the CTAs below.
    monkeypatch.setattr(Grid, "below", lambda self, c, it, n: iter(()))
    faults(lambda: Grid(3), "learned fused")
