"""The training kernels (train.cuh) at their edges: nodes short of, at and past a
step of 16, rows whose entries do not fit the step's shared memory (224), rows of
uneven length, all probe recipes. Tolerances as in test_gpu_learned.py: BF16
activations round at the same points as the oracle's, sums in another order.
"""
import numpy as np
import pytest

import cgxx_b200 as cg
from cgxx_b200 import generators as G
from conftest import random_crs
from oracle import gnn_oracle as GO

pytestmark = pytest.mark.gpu


def _params(seed):
    p = GO.init_params(seed)
    return (p + 0.05 * np.random.default_rng(seed + 100).standard_normal(p.size)).astype(np.float32)


def _diag(n):
    return G.Crs(n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32),
                 np.linspace(1.0, 2.0, n))


CASES = [("diag_1", lambda: _diag(1)), ("diag_16", lambda: _diag(16)),
         ("poisson_4", lambda: G.poisson2d(4)),
         ("random_17", lambda: random_crs(17, 0, 6, seed=3, spd=True)),
         ("random_63", lambda: random_crs(63, 0, 10, seed=4, spd=True)),
         ("long_rows_130", lambda: random_crs(130, 0, 60, seed=5, spd=True)),
         ("graph_700", lambda: G.geometric_graph(700, seed=6))]


@pytest.mark.parametrize("name,make", CASES, ids=[c[0] for c in CASES])
def test_gradient_at_the_edges(name, make):
    A = make()
    params = _params(11)
    V = np.random.default_rng(1).choice([-1.0, 1.0], size=(A.N, 8)).astype(np.float32)
    with cg.Handle(0) as h:
        h.upload_crs(A.ptr, A.index, A.value)
        h.learned_setup()
        net = cg.Gnn(0, params)
        loss, grad = net.loss_grad(h, probes=V)
        again = net.loss_grad(h, probes=V)
        net.close()
    lo, go = GO.loss_and_grad(GO.Graph(A.ptr, A.index, A.value), params, V)
    assert abs(loss - lo) <= 1e-3 * abs(lo)
    assert np.linalg.norm(grad - go) <= 3e-2 * np.linalg.norm(go)
    assert again[0] == loss and np.array_equal(again[1], grad)


def test_gradient_past_the_largest_numbers():
    """One node whose last layer's gradient is infinite in all features but two: one
    that rounds to infinity in BF16 only, one ordinary. The last layer's weight
    gradients are what FP32 gives: infinite, and finite there (the products of two
    FP32 numbers, 2^-20 apart from the oracle's at most).

    W_in = W_l = 0 and biases of 2^-126 give h = 2^-126, 2 and 3 times that into the
    last layer and 2^-124 out of it; the head reads only the diagonal's output."""
    A = _diag(1)
    tiny = 2.0 ** -126
    P = {n: np.zeros(s) for n, s in GO.param_shapes()}
    for name in ("b_in", "b_0", "b_1", "b_2"):
        P[name][:] = tiny
    P["W_h"][1] = 2.0 ** 125
    g = 30 * 2.0 + GO.DIAG_OFFSET  # the factor's entry; softplus adds nothing here
    dO = 4.0 * (g * g - 1.0) * g
    P["W_h"][1, 0], P["W_h"][1, 1] = 3.4e38 / dO, 1e30 / dO
    params = np.concatenate([P[n].ravel() for n, _ in GO.param_shapes()]).astype(np.float32)
    V = np.ones((1, 8), np.float32)
    with cg.Handle(0) as h:
        h.upload_crs(A.ptr, A.index, A.value)
        h.learned_setup()
        net = cg.Gnn(0, params)
        grad = net.loss_grad(h, probes=V)[1]
        net.close()
    want = GO.loss_and_grad(GO.Graph(A.ptr, A.index, A.value), params, V)[1]
    got, ref = (GO.unflatten(v)["W_2"][:, :GO.WIDTH] for v in (grad, want))
    assert np.isfinite(ref[:2]).all() and np.isinf(ref[2:]).all()
    assert 3.3962e38 * 3 * tiny < ref[0, 0] < 3.4028e38 * 3 * tiny
    np.testing.assert_allclose(got, ref, rtol=2.0 ** -20)
