"""The persistent solves as one thread-block cluster, on both sides of the sizes
where the form, the CTA width or the cluster size changes, against the loops of
single kernels. The rows' sums are the same, the dot products' order differs:
iteration counts agree to 2 % + 2; at a residual of 1e-12 the solutions differ by at
most 1e-12 times the condition number (below 1e5 here) times 10.
"""
import numpy as np
import pytest

import cgxx_b200 as cg
from cgxx_b200 import generators as G
from cgxx_b200 import learned as LRN

pytestmark = pytest.mark.gpu

FAMILIES = {"poisson": G.poisson2d, "diff7": lambda n: G.diffusion3d(n, 7, corr_len=3.0, seed=1),
            "diff27": lambda n: G.diffusion3d(n, 27, corr_len=3.0, seed=2),
            "graph": lambda n: G.geometric_graph(n, seed=3)}
CASES = [("poisson", n) for n in (16, 17, 32, 64, 65, 91, 128, 129)] + \
        [("diff7", n) for n in (7, 16, 20, 25)] + [("diff27", n) for n in (7, 16, 20, 21)] + \
        [("graph", n) for n in (256, 257, 4097, 8192, 8193)]


def _solve(h, loop, **kw):
    h.fill_vector("X", 0.0)
    r = h.solve(loop=loop, max_iterations=20000, **kw)
    assert r["converged"] and r["fell_back"] == 0
    return r["iterations"], h.get_vector("X")


@pytest.mark.parametrize("family,n", CASES)
def test_cluster_matches_single_kernels(family, n):
    A = FAMILIES[family](n)
    k = A.matvec(np.random.default_rng(4).uniform(-1, 1, A.N))
    with cg.Handle(0) as h:
        h.upload_crs(A.ptr, A.index, A.value)
        h.jacobi_from_matrix()
        h.set_vector("K", k)
        a, xa = _solve(h, cg.LOOP_GRAPH, tolerance=1e-12)
        b, xb = _solve(h, cg.LOOP_CHUNKED, tolerance=1e-12)
        assert abs(a - b) <= 0.02 * b + 2
        assert np.linalg.norm(xa - xb) <= 1e-6 * np.linalg.norm(xb)
        net = None
        for pc in (cg.PRECOND_JACOBI, cg.PRECOND_LEARNED):
            if pc == cg.PRECOND_LEARNED:
                if family == "poisson":
                    continue
                net = cg.Gnn(0, LRN.load_weights(LRN.DEFAULT_WEIGHTS)[0])
                h.learned_setup()
                h.learned_factor(net, 1e-4)
            kw = dict(tolerance=1e-10, precision=cg.PRECISION_MIXED, preconditioner=pc)
            a, xa = _solve(h, cg.LOOP_GRAPH, **kw)
            b, _ = _solve(h, cg.LOOP_KERNELS, **kw)
            assert abs(a - b) <= 0.02 * b + 2
            assert np.linalg.norm(k - A.matvec(xa)) <= 1e-10 * np.linalg.norm(k)
        if net:
            net.close()
