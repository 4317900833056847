"""Inner solves on FP32 values by offset (offsets.cuh, OffsetPhases): 27-point grids
around the tile widths, against the loop of per-iteration kernels
on SELL-U. The products add the same values in the same order; the dot products'
order differs, so the inner counts agree to 2 % + 2 and both solutions reach the
FP64 residual. Values that are not symmetric in FP32 leave the form.
"""
import numpy as np
import pytest

import cgxx_b200 as cg
from cgxx_b200 import generators as G

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _solve(h, loop, k):
    h.set_vector("K", k)
    h.fill_vector("X", 0.0)
    r = h.solve(max_iterations=20000, tolerance=TOL, precision=cg.PRECISION_MIXED, loop=loop)
    return r, h.get_vector("X")


@pytest.mark.parametrize("n", [3, 5, 11, 32, 53, 55])
def test_inner_solves_by_offset(n):
    A = G.diffusion3d(n, 27, sigma=1.0, corr_len=3.0, seed=7)
    k = A.matvec(np.random.default_rng(1).uniform(-1, 1, A.N))
    with cg.Handle(0) as h:
        h.upload_crs(A.ptr, A.index, A.value)
        h.jacobi_from_matrix()
        a, xa = _solve(h, cg.LOOP_GRAPH, k)
        b, xb = _solve(h, cg.LOOP_KERNELS, k)
        assert a["inner_form"] == 3 and a["converged"] and b["converged"]
        assert abs(a["iterations"] - b["iterations"]) <= 0.02 * b["iterations"] + 2
        for x in (xa, xb):
            assert np.linalg.norm(k - A.matvec(x)) <= TOL * np.linalg.norm(k)
        # One value off by 1e-4: no longer symmetric, still solved (to 1e-10 of a
        # matrix 1e-4 away from symmetric, by refinement).
        v = A.value.copy()
        j = int(A.ptr[1]) - 1
        v[j] *= 1.0 + 1e-4
        B = G.Crs(A.N, A.ptr, A.index, v)
        h.update_crs_values(v)
        h.jacobi_from_matrix()
        c, xc = _solve(h, cg.LOOP_GRAPH, k)
        assert c["converged"]
        assert np.linalg.norm(k - B.matvec(xc)) <= TOL * np.linalg.norm(k)
