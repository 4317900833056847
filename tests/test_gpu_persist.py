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


def fp64_matrix(kind, N):
    """Matrices of each form the plain persistent solve stores, and two that
    it must leave to the rows."""
    if kind == "half3":  # up to 3 non-negative offsets
        return band_matrix(N, (1, 61))
    if kind == "half4":
        return band_matrix(N, (1, 61, 1777))
    if kind == "half14":
        A = band_matrix(N, (1, 2, 31, 32, 33, 901, 931, 932, 933, 962, 963, 964, 965))
        A.value[A.rows() == A.index] += 20.0
        return A
    A = band_matrix(N, (1, 61, 1777) if kind in ("all7", "reversed")
                    else (1, 2, 31, 32, 33, 901, 931, 932, 933, 962, 963, 964, 965))
    if kind == "all27":
        A.value[A.rows() == A.index] += 20.0
    if kind in ("all7", "all27") and A.nz > A.N:
        # Not symmetric in the last bit of one entry: every offset is stored.
        k = np.flatnonzero(A.rows() != A.index)[0]
        A.value[k] = np.nextafter(A.value[k], 0.0)
    if kind == "reversed":  # columns descend: not the order of the offsets
        order = np.lexsort((-A.index, A.rows()))
        A = G.Crs(A.N, A.ptr, A.index[order].copy(), A.value[order].copy())
    if kind == "sparse":  # 27 offsets, most of them empty
        keep = (A.rows() == A.index) | ((A.rows() + A.index) % 16 == 0)
        rows, cols, vals = A.rows()[keep], A.index[keep], A.value[keep]
        A = G.crs_from_unsorted(N, rows, cols, vals)
    return A


KINDS = ["half3", "half4", "half14", "all7", "all27", "reversed", "sparse"]


def upload(handle, A, fmt):
    if fmt == "ell":
        handle.upload_ell(A.N, A.nz, *G.to_ell(A))
    elif fmt == "coo":
        handle.upload_coo(A.N, A.rows(), A.index, A.value)
    else:
        handle.upload_crs(A.ptr, A.index, A.value)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("N", [1, 2, 33, 255, 257, 1025, 4098, 37889, 75777, 151553])
def test_plain_forms_agree_with_the_kernels(handle, kind, N):
    """Ten iterations of every form against the chunked kernels. The forms
    differ in the order of the dot products' sums only: a relative error of at
    most N * 2^-53 in each, 20 of them, and as the iterates depend smoothly on
    the scalars (condition at most 7), at most 20 * 7 * N * 2^-53 in x."""
    A = fp64_matrix(kind, N)
    b, _ = G.rhs_for(A, seed=3)
    fmt = ("crs", "ell", "coo")[(N + len(kind)) % 3]
    upload(handle, A, fmt)
    handle.jacobi_from_matrix()
    handle.set_vector("K", b)
    for pc in (cg.PRECOND_JACOBI, cg.PRECOND_NONE):
        out = {}
        for loop in (cg.LOOP_CHUNKED, cg.LOOP_GRAPH, cg.LOOP_PERSISTENT,
                     cg.LOOP_PERSISTENT_SPLIT):
            handle.fill_vector("X", 0.25)
            r = handle.solve(max_iterations=10, tolerance=1e-30, preconditioner=pc, loop=loop)
            out[loop] = (r, [handle.get_vector(v) for v in "XRPQ"])
        r0, v0 = out[cg.LOOP_CHUNKED]
        if not np.isfinite(v0[0]).all() or r0["residual"] < 1e-12:
            continue  # converged to zero: the last iterates are rounding noise
        bound = 20 * KAPPA * N * 2.0 ** -53
        for loop in (cg.LOOP_GRAPH, cg.LOOP_PERSISTENT, cg.LOOP_PERSISTENT_SPLIT):
            r, v = out[loop]
            assert r["iterations"] == r0["iterations"] == 10, (loop, r)
            assert r["converged"] == 0
            for name, a, c in zip("XRPQ", v, v0):
                scale = max(np.linalg.norm(c), np.linalg.norm(v0[0]) * 1e-3)
                assert np.linalg.norm(a - c) <= bound * scale + 1e-300, (loop, pc, name)


@pytest.mark.parametrize("loop", [cg.LOOP_GRAPH, cg.LOOP_PERSISTENT, cg.LOOP_PERSISTENT_SPLIT])
def test_plain_forms_stop_as_the_kernels_do(handle, loop):
    """Convergence, the iteration limit, a NaN that never converges, and new
    values on the same pattern."""
    A = band_matrix(5003, (1, 61, 1777))
    b, xs = G.rhs_for(A, seed=4)
    handle.upload_crs(A.ptr, A.index, A.value)
    handle.jacobi_from_matrix()
    handle.set_vector("K", b)
    want = {}
    for lp in (cg.LOOP_CHUNKED, loop):
        handle.fill_vector("X", 0.0)
        r = handle.solve(max_iterations=1000, tolerance=1e-11, loop=lp)
        want[lp] = r["iterations"]
        assert r["converged"] == 1 and r["residual"] <= 1e-11
        assert np.linalg.norm(handle.get_vector("X") - xs) <= 1e-11 * KAPPA * np.linalg.norm(xs)
    assert want[loop] == want[cg.LOOP_CHUNKED]
    handle.fill_vector("X", 0.0)
    r = handle.solve(max_iterations=1, tolerance=1e-11, loop=loop)
    assert r["iterations"] == 1 and r["converged"] == 0
    v = 3.0 * A.value
    handle.update_crs_values(v)
    handle.jacobi_from_matrix()
    handle.fill_vector("X", 0.0)
    r = handle.solve(max_iterations=1000, tolerance=1e-11, loop=loop)
    assert r["converged"] == 1
    assert np.linalg.norm(3.0 * handle.get_vector("X") - xs) <= 1e-11 * KAPPA * np.linalg.norm(xs)
    bad = b.copy()
    bad[17] = np.nan
    handle.set_vector("K", bad)
    handle.fill_vector("X", 0.0)
    r = handle.solve(max_iterations=7, tolerance=1e-11, loop=loop)
    assert r["iterations"] == 7 and r["converged"] == 0


@pytest.mark.parametrize("kind,N", [("half4", 729001), ("all7", 1048577), ("half3", 1199999),
                                    ("half4", 1200001), ("reversed", 884736)])
def test_plain_default_takes_a_persistent_form(handle, kind, N):
    """0.7M to 1.2M rows and at most seven offsets: ten iterations of the default
    loop agree with the chunked kernels (the bound of
    test_plain_forms_agree_with_the_kernels) and take less time; the default loop
    run as those kernels takes as long as they do."""
    A = fp64_matrix(kind, N)
    b, _ = G.rhs_for(A, seed=3)
    upload(handle, A, "coo" if kind == "reversed" else ("crs", "ell")[N % 2])
    handle.jacobi_from_matrix()
    handle.set_vector("K", b)
    x, ms = {}, {}
    for loop in (cg.LOOP_CHUNKED, cg.LOOP_GRAPH):
        for _ in range(4):  # the first includes the layout
            handle.fill_vector("X", 0.25)
            r = handle.solve(max_iterations=10, tolerance=1e-30, loop=loop)
            assert r["iterations"] == 10
            ms[loop] = min(ms.get(loop, 1e9), r["solve_ms"])
        x[loop] = handle.get_vector("X")
    want = x[cg.LOOP_CHUNKED]
    assert np.linalg.norm(x[cg.LOOP_GRAPH] - want) <= \
        20 * KAPPA * N * 2.0 ** -53 * np.linalg.norm(want)
    assert ms[cg.LOOP_GRAPH] < 0.8 * ms[cg.LOOP_CHUNKED], ms


def test_solve_ms_leaves_out_the_layout():
    """The first plain solve on a matrix reports what the next ones do, up to a tenth
    and 0.1 ms: its layout (allocations, two passes over A, waits for the host) is not
    the solve. Another handle has loaded the kernels before."""
    A = G.diffusion3d(128, 7, corr_len=4.0, seed=1)
    for _ in range(2):
        with cg.Handle(0) as h:
            h.upload_crs(A.ptr, A.index, A.value)
            h.jacobi_from_matrix()
            h.fill_vector("K", 1.0)
            ms = []
            for _ in range(4):
                h.fill_vector("X", 0.0)
                h.synchronize()
                ms.append(h.solve(max_iterations=10, tolerance=1e-30)["solve_ms"])
    assert ms[0] <= 1.1 * min(ms[1:]) + 0.1, ms
