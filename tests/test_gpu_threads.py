"""Several host threads with a handle each: their solves of different sizes run the
same kernels with different amounts of shared memory, and give, bit for bit, what
they give alone."""
import threading

import numpy as np
import pytest

import cgxx_b200 as cg
from cgxx_b200 import generators as G
from conftest import random_crs

pytestmark = pytest.mark.gpu

# Two matrices whose solves share a kernel: by offset in FP64, on the FP32 band, and
# the loop of single kernels with CRS tiles of about 900 and 1700 entries.
GRIDS = [lambda: G.diffusion3d(34, 7, corr_len=3.0, seed=1),
         lambda: G.diffusion3d(79, 7, corr_len=3.0, seed=2)]
ROWS = [lambda: random_crs(20000, max_len=40, seed=3, spd=True),
        lambda: random_crs(50000, max_len=90, seed=4, spd=True)]
PAIRS = {
    "persistent": (GRIDS, dict(loop=cg.LOOP_GRAPH)),
    "inner": (GRIDS, dict(loop=cg.LOOP_GRAPH, precision=cg.PRECISION_MIXED)),
    "crs": (ROWS, dict(loop=cg.LOOP_KERNELS)),
}


@pytest.mark.parametrize("name", PAIRS)
def test_concurrent_solves_give_what_they_give_alone(name):
    matrices, options = PAIRS[name]
    systems = []
    for make in matrices:
        A = make()
        h = cg.Handle(0)
        h.upload_crs(A.ptr, A.index, A.value)
        h.jacobi_from_matrix()
        h.set_vector("K", np.random.default_rng(5).uniform(-1, 1, A.N))
        systems.append(h)

    def solve(h):
        h.fill_vector("X", 0.0)
        h.solve(max_iterations=12, tolerance=1e-13, **options)
        return h.get_vector("X")

    alone = [solve(h) for h in systems]
    failed = []

    def work(h, want):
        try:
            for _ in range(300):
                assert np.array_equal(solve(h), want)
        except Exception as e:  # a thread's failure is the test's
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(systems, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for h in systems:
        h.close()
    assert not failed, failed
