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
