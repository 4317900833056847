"""Persistent FP64 solves on sorted slices (slices.cuh) against the chunked loop of
the CRS kernels, on matrices that no by-offset form holds. A row's products are
added in the same order, so q = A p of the first iteration is bit-identical; the
dot products' order differs, so later iterates agree to rounding: the solutions at
a residual of 1e-11 differ by at most 1e-11 times the condition number, which is
below 1e2 for these diagonally dominant matrices (1e-8 with a margin of 10).
"""
import numpy as np
import pytest

import cgxx_b200 as cg
from cgxx_b200 import generators as G
from cgxx_b200 import learned as LRN
from conftest import random_crs

pytestmark = pytest.mark.gpu


def _dense_row(N, extra, seed):
    """random_crs plus a symmetric first row and column of `extra` entries."""
    A = random_crs(N, 0, 8, seed=seed, spd=True)
    rows = np.repeat(np.arange(N), np.diff(A.ptr))
    j = np.arange(1, extra + 1)
    d = np.zeros(N)
    d[0], d[1:extra + 1] = 0.01 * extra, 0.01
    rows = np.concatenate([rows, np.zeros(extra, int), j, np.arange(N)])
    cols = np.concatenate([A.index, j, np.zeros(extra, int), np.arange(N)])
    vals = np.concatenate([A.value, np.full(2 * extra, -0.01), d + 1e-3])
    key = rows.astype(np.int64) * N + cols
    uk, inv = np.unique(key, return_inverse=True)
    return G.crs_from_unsorted(N, uk // N, uk % N, np.bincount(inv, weights=vals))


def _shuffled(A, seed):
    """The same matrix, each row's entries in another order."""
    rng = np.random.default_rng(seed)
    index, value = A.index.copy(), A.value.copy()
    for i in range(A.N):
        s = slice(A.ptr[i], A.ptr[i + 1])
        o = rng.permutation(A.ptr[i + 1] - A.ptr[i])
        index[s], value[s] = index[s][o], value[s][o]
    return G.Crs(A.N, A.ptr, index, value)


CASES = [
    ("random_33", lambda: random_crs(33, 0, 12, seed=1, spd=True)),
    ("random_255", lambda: random_crs(255, 0, 20, seed=2, spd=True)),
    ("random_1500", lambda: random_crs(1500, 0, 40, seed=3, spd=True)),
    ("shuffled_3000", lambda: _shuffled(random_crs(3000, 0, 20, seed=4, spd=True), 5)),
    ("graph_40001", lambda: G.geometric_graph(40001, seed=6)),   # 512-thread CTAs
    ("graph_160001", lambda: G.geometric_graph(160001, seed=7)),  # 1024, two steps
    ("dense_row_2000", lambda: _dense_row(2000, 1500, 8)),
    ("row_of_5000", lambda: _dense_row(6000, 5000, 9)),  # too long: stays on the graph
]


@pytest.mark.parametrize("fmt", ["crs", "coo"])
@pytest.mark.parametrize("name,make", CASES, ids=[c[0] for c in CASES])
def test_solve_matches_the_chunked_loop(name, make, fmt):
    A = make()
    rng = np.random.default_rng(10)
    k = rng.standard_normal(A.N)
    x0 = rng.standard_normal(A.N)
    jac = name != "random_255"
    pc = cg.PRECOND_JACOBI if jac else cg.PRECOND_NONE
    with cg.Handle(0) as h:
        if fmt == "crs":
            h.upload_crs(A.ptr, A.index, A.value)
        else:
            h.upload_coo(A.N, np.repeat(np.arange(A.N), np.diff(A.ptr)).astype(np.int32), A.index,
                         A.value)
        h.jacobi_from_matrix()
        h.set_vector("K", k)

        def solve(loop, **kw):
            h.set_vector("X", x0)
            r = h.solve(loop=loop, preconditioner=pc, **kw)
            return r, {v: h.get_vector(v) for v in "XRPQ"}

        _, one = solve(cg.LOOP_GRAPH, max_iterations=1, tolerance=1e-300)
        _, ref1 = solve(cg.LOOP_CHUNKED, max_iterations=1, tolerance=1e-300)
        assert np.array_equal(one["Q"], ref1["Q"])
        for v in "XRP":
            assert np.allclose(one[v], ref1[v], rtol=0, atol=1e-13 * np.abs(ref1[v]).max())
        a, va = solve(cg.LOOP_GRAPH, max_iterations=2000, tolerance=1e-11)
        b, vb = solve(cg.LOOP_CHUNKED, max_iterations=2000, tolerance=1e-11)
        assert a["converged"] and b["converged"]
        assert abs(a["iterations"] - b["iterations"]) <= 1 + 0.02 * b["iterations"]
        # Graphs (shift 1e-3) are worse conditioned than the random matrices.
        bound = 1e-5 if name.startswith("graph") else 1e-8
        assert np.linalg.norm(va["X"] - vb["X"]) <= bound * np.linalg.norm(vb["X"])
        # New values of the same pattern reach the slices.
        if fmt == "crs":
            h.update_crs_values(2.0 * A.value)
            h.jacobi_from_matrix()
            c, vc = solve(cg.LOOP_GRAPH, max_iterations=2000, tolerance=1e-11)
            assert c["converged"]
            assert np.linalg.norm(2.0 * vc["X"] - vb["X"]) <= bound * np.linalg.norm(vb["X"])


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("name,make", CASES[:7], ids=[c[0] for c in CASES[:7]])
def test_inner_solves_match_the_kernels(name, make, learned):
    """Mixed solves on the FP32 and BF16 slices against the loop of per-iteration
    kernels (CRS and SELL-U): the same products in the same order, so the inner
    counts agree to 2 % + 2 and both reach the FP64 residual. The second solve is
    on new values with a new factor."""
    A = make()
    rng = np.random.default_rng(12)
    k = A.matvec(rng.uniform(-1, 1, A.N))
    tol = 1e-10
    with cg.Handle(0) as h:
        h.upload_crs(A.ptr, A.index, A.value)
        net = cg.Gnn(0, LRN.load_weights(LRN.DEFAULT_WEIGHTS)[0])
        for scale in (1.0, 2.0):
            h.update_crs_values(scale * A.value)
            h.jacobi_from_matrix()
            pc = cg.PRECOND_JACOBI
            if learned:
                h.learned_setup()
                h.learned_factor(net, 1e-4)
                pc = cg.PRECOND_LEARNED
            h.set_vector("K", scale * k)
            its = {}
            for loop in (cg.LOOP_GRAPH, cg.LOOP_KERNELS):
                h.fill_vector("X", 0.0)
                r = h.solve(max_iterations=20000, tolerance=tol, loop=loop, preconditioner=pc,
                            precision=cg.PRECISION_MIXED)
                assert r["converged"] and r["fell_back"] == 0
                if loop == cg.LOOP_GRAPH and name in ("graph_40001", "graph_160001"):
                    assert r["inner_form"] == 3
                x = h.get_vector("X")
                assert np.linalg.norm(k - A.matvec(x)) <= tol * np.linalg.norm(k)
                its[loop] = r["iterations"]
            assert abs(its[cg.LOOP_GRAPH] - its[cg.LOOP_KERNELS]) <= 0.02 * its[cg.LOOP_KERNELS] + 2
        net.close()


def test_rejected_slices_keep_no_memory():
    """Eight rows of 200 entries among every 1024 of one: the slices would more than
    double the entries, so the solve stays on the rows and what was laid out on the
    way (48 bytes a row) is given back. Kernels and graphs are loaded by a small
    solve first; they and the flags may take a tenth of those bytes."""
    import torch

    def solve(N):
        rows = np.arange(0, N, 128)
        r = np.concatenate([np.arange(N), np.repeat(rows, 199)])
        c = np.concatenate([np.arange(N), (rows[:, None] + 31 * np.arange(1, 200)).ravel() % N])
        A = G.crs_from_unsorted(N, r, c, np.where(r == c, 4.0, 1e-3))
        h = cg.Handle(0)
        h.upload_crs(A.ptr, A.index, A.value)
        h.fill_vector("K", 1.0)
        h.synchronize()
        free = torch.cuda.mem_get_info()[0]
        h.solve(max_iterations=5, tolerance=1e-30, preconditioner=cg.PRECOND_NONE)
        taken = free - torch.cuda.mem_get_info()[0]
        h.close()
        return taken

    solve(20000)
    N = 2000000
    assert solve(N) <= 48 * N / 10
