"""The persistent solves at the edges of their CTA shapes, against the
per-iteration kernels (the KERNELS and CHUNKED loop modes).

The matrices have 8 on the diagonal and -1 at up to six offsets, so by
Gershgorin their eigenvalues lie in [2, 14]. Two solutions whose relative
residuals are at most tol then differ by at most 2 * tol * 14 / 2 of their norm.
"""
import numpy as np
import pytest

import cgxx_b200 as cg
from cgxx_b200 import generators as G
from cgxx_b200 import learned as LRN

pytestmark = pytest.mark.gpu

KAPPA = 7.0


def band_matrix(N, offsets):
    """Symmetric, 8 on the diagonal, -1 at +-offsets (those below N)."""
    i = np.arange(N, dtype=np.int64)
    rows, cols, vals = [i], [i], [np.full(N, 8.0)]
    for d in offsets:
        if d < N:
            lo = i[d:]
            rows += [lo, lo - d]
            cols += [lo - d, lo]
            vals += [np.full(N - d, -1.0)] * 2
    return G.crs_from_unsorted(N, np.concatenate(rows), np.concatenate(cols),
                               np.concatenate(vals))


# Rows around one thread, warp, quad, CTA width (256, 512, 1024), the bounds
# 148 * 256 and 200000 of the CTA shapes, and a last tile with a ragged end;
# offsets from the next row to several CTAs away.
SIZES = [1, 2, 3, 5, 33, 255, 257, 1023, 1025, 4098, 37887, 37889, 75777, 199999, 200003,
         151553]


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("N", SIZES)
def test_mixed_forms_agree_with_the_kernels(handle, N, learned):
    tol = 1e-9
    A = band_matrix(N, (1, 37, 1501))
    b, _ = G.rhs_for(A, seed=N)
    handle.upload_crs(A.ptr, A.index, A.value)
    handle.upload_jacobi(1.0 / A.diagonal())
    handle.set_vector("K", b)
    pc = cg.PRECOND_JACOBI
    if learned:
        handle.learned_setup()
        net = cg.Gnn(0, LRN.load_weights(LRN.DEFAULT_WEIGHTS)[0])
        handle.learned_factor(net, 1e-4)
        net.close()
        pc = cg.PRECOND_LEARNED
    out = {}
    for loop in (cg.LOOP_KERNELS, cg.LOOP_GRAPH, cg.LOOP_PERSISTENT, cg.LOOP_PERSISTENT_SPLIT):
        handle.fill_vector("X", 0.0)
        r = handle.solve(max_iterations=2000, tolerance=tol, preconditioner=pc,
                         precision=cg.PRECISION_MIXED, loop=loop)
        assert r["converged"] == 1 and r["fell_back"] == 0, (loop, r)
        out[loop] = (r["iterations"], handle.get_vector("X"))
    its, x = out[cg.LOOP_KERNELS]
    for loop in (cg.LOOP_GRAPH, cg.LOOP_PERSISTENT, cg.LOOP_PERSISTENT_SPLIT):
        assert abs(out[loop][0] - its) <= 2, (loop, out[loop][0], its)
        assert np.linalg.norm(out[loop][1] - x) <= 2 * tol * KAPPA * np.linalg.norm(x), loop


@pytest.mark.parametrize("N", [1025, 151551, 151553, 303110])
@pytest.mark.parametrize("learned", [False, True])
def test_sell_form_agrees_with_the_kernels(handle, N, learned):
    """Ten offsets (no band): the SELL-U form with 512- and 1024-thread CTAs."""
    tol = 1e-9
    A = band_matrix(N, (1, 2, 3))
    B = band_matrix(N, (31, 977))
    v = A.value.copy()
    v[A.rows() == A.index] += 4.0  # room for the two further offsets
    rows = np.concatenate([A.rows(), B.rows()[B.rows() != B.index]])
    cols = np.concatenate([A.index, B.index[B.rows() != B.index]])
    M = G.crs_from_unsorted(N, rows, cols,
                            np.concatenate([v, B.value[B.rows() != B.index]]))
    b, _ = G.rhs_for(M, seed=N)
    handle.upload_crs(M.ptr, M.index, M.value)
    handle.upload_jacobi(1.0 / M.diagonal())
    handle.set_vector("K", b)
    pc = cg.PRECOND_JACOBI
    if learned:
        handle.learned_setup()
        net = cg.Gnn(0, LRN.load_weights(LRN.DEFAULT_WEIGHTS)[0])
        handle.learned_factor(net, 1e-4)
        net.close()
        pc = cg.PRECOND_LEARNED
    out = {}
    for loop in (cg.LOOP_KERNELS, cg.LOOP_GRAPH):
        handle.fill_vector("X", 0.0)
        r = handle.solve(max_iterations=2000, tolerance=tol, preconditioner=pc,
                         precision=cg.PRECISION_MIXED, loop=loop)
        assert r["converged"] == 1 and r["fell_back"] == 0, (loop, r)
        out[loop] = (r, handle.get_vector("X"))
    assert out[cg.LOOP_GRAPH][0]["inner_form"] == 3
    assert abs(out[cg.LOOP_GRAPH][0]["iterations"] - out[cg.LOOP_KERNELS][0]["iterations"]) <= 2
    x = out[cg.LOOP_KERNELS][1]
    # 12 on the diagonal, five offsets: eigenvalues in [2, 22].
    assert np.linalg.norm(out[cg.LOOP_GRAPH][1] - x) <= 2 * tol * 11 * np.linalg.norm(x)
