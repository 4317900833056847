"""The gradient's precision: each parameter block against 64-bit arithmetic with the
same BF16 rounding points.

The weights up to the last layer are multiples of 1/16 and the scaled 5-point matrix
has entries of 1/4, so every sum of the forward pass up to the head is exact in FP32:
both sides round the same numbers to BF16, and what is left is the rounding of FP32
sums behind it. In FP32 on the CPU that is 9e-8 to 5.5e-7 of a block's norm on these
matrices; the device adds in another order and calls CUDA's expf and log1pf, hence
2e-6. A backward pass that kept the layers' gradients in BF16 would be off by 4e-5 or
more (test_gradients_in_bf16_would_show).
"""
import numpy as np
import pytest
import torch

import cgxx_b200 as cg
from cgxx_b200 import generators as G
from oracle import gnn_oracle as GO

TOLERANCE = 2e-6
CASES = [(n, seed) for n in (3, 4, 7, 17, 33) for seed in (1, 2)]


def problem(n, seed):
    rng = np.random.default_rng(seed)
    P = {}
    for name, shape in GO.param_shapes():
        if name in ("W_h", "b_h"):
            P[name] = rng.normal(0, 0.1, shape)
        elif name in ("W_0", "W_1", "W_2", "b_0", "b_1", "b_2"):
            P[name] = rng.integers(-2, 3, shape) / 16.0
        else:
            P[name] = rng.integers(-4, 5, shape) / 8.0
    P["W_in"][:, 2] = 0.0  # its feature, a sixth of the degree, is not dyadic
    params = np.concatenate([P[k].ravel() for k, _ in GO.param_shapes()]).astype(np.float32)
    A = G.poisson2d(n)
    return A, params, rng.choice([-1.0, 1.0], size=(A.N, 8)).astype(np.float32)


class Bf16Gradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, grad):
        return grad.to(torch.bfloat16).to(grad.dtype)


def gradient64(A, params, V, monkeypatch=None):
    """The oracle's gradient in 64 bits; with monkeypatch, each layer's
    pre-activation gradients rounded to BF16."""
    g = GO.Graph(A.ptr, A.index, A.value)
    for name in ("ah", "ow", "lw", "feat"):
        setattr(g, name, getattr(g, name).double())
    flat = torch.tensor(params, dtype=torch.float64, requires_grad=True)
    if monkeypatch:
        relu = torch.relu
        monkeypatch.setattr(torch, "relu", lambda x: relu(Bf16Gradient.apply(x)))
    gdiag, goff = GO.forward(g, flat)
    GO.loss(g, gdiag, goff, torch.tensor(V, dtype=torch.float64)).backward()
    return flat.grad.numpy()


def block_errors(grad, want):
    got, ref = GO.unflatten(np.asarray(grad, np.float64)), GO.unflatten(want)
    return {k: np.linalg.norm(got[k] - ref[k]) / np.linalg.norm(ref[k]) for k in ref}


@pytest.mark.gpu
@pytest.mark.parametrize("n,seed", CASES)
def test_gradient_is_fp32_exact(n, seed):
    A, params, V = problem(n, seed)
    with cg.Handle(0) as h:
        h.upload_crs(A.ptr, A.index, A.value)
        h.learned_setup()
        net = cg.Gnn(0, params)
        grad = net.loss_grad(h, probes=V)[1]
        net.close()
    errors = block_errors(grad, gradient64(A, params, V))
    assert max(errors.values()) <= TOLERANCE, errors


@pytest.mark.parametrize("n,seed", CASES)
def test_gradients_in_bf16_would_show(n, seed, monkeypatch):
    A, params, V = problem(n, seed)
    want = gradient64(A, params, V)
    errors = block_errors(gradient64(A, params, V, monkeypatch), want)
    layers = [errors[k] for k in ("W_in", "b_in", "W_0", "b_0", "W_1", "b_1", "W_2", "b_2")]
    assert min(layers) > 10 * TOLERANCE, errors
