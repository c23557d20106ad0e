"""The fused inference kernel at the edges of its 128-row tiles and of its grid (152 CTAs), every row against the layer-wise
forward of the same network and a sample against FP64 on the BF16 weights.

Bound: a layer keeps its input to 2^-17 and its sums to 2^-18 of their magnitude, both random from term to term: seven
layers of 1.1e-5 each, 8e-5 of the largest output; 1e-4 is asserted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("n", [1, 127, 128, 129, 256 * 3 + 1, SMS * 128 - 1, SMS * 128, SMS * 128 + 1, 2 * SMS * 128 + 1,
                               3 * SMS * 128 + 77])
@pytest.mark.parametrize("shift", [0, 1])
def test_every_row(n, shift):
    import torch
    from sgl_analytic_gb300 import surrogate as S
    from sgl_analytic_gb300._lib import Engine
    eng = Engine(0)
    mlp = S.MLP(eng, width=256, depth=6, seed=11)
    with torch.cuda.stream(mlp.stream):
        for i, b in enumerate(mlp.b):
            b += 0.1 * torch.cos(torch.arange(b.numel(), device="cuda") + i)
    rng = np.random.default_rng(n + shift)
    X = rng.uniform(-1.7, 1.7, (n, 8)).astype(np.float32)
    (flat,) = S.to_device(eng, np.concatenate([np.zeros(shift, np.float32), X.ravel()]))
    Xd = flat[shift:].view(n, 8)                               # the rows start `shift` floats into an allocation
    Y, F = mlp.infer(Xd), mlp.forward(Xd)
    mlp.stream.synchronize()
    Y, F = Y.double().cpu().numpy(), F.double().cpu().numpy()
    assert Y.shape == (n, 2)
    rows = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n)]))
    A = X[rows].astype(np.float64)
    for l, (w, b) in enumerate(zip(mlp.W, mlp.b)):
        A = A @ w.bfloat16().double().cpu().numpy() + b.double().cpu().numpy()
        if l < len(mlp.W) - 1:
            A = A / (1.0 + np.exp(-A))
    top = np.max(np.abs(A))
    assert top > 0.05                                          # there is something to compare
    assert np.max(np.abs(Y - F)) <= 1e-4 * top
    assert np.max(np.abs(Y[rows] - A)) <= 1e-4 * top
