"""The fused inference kernel of the surrogate MLP at the edges of its 128-row tiles and of its grid, against
the network in FP64 with the BF16 weights the kernel uses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 152
EPS = 2.0 ** -24


@pytest.fixture(scope="module")
def eng():
    from sgl_analytic_gb300._lib import Engine
    return Engine(0)


def _bf16(W):
    import torch
    return torch.from_numpy(W).to(torch.bfloat16).to(torch.float64).numpy()


def _exact_and_bound(W, b, X):
    """The network in FP64 and a bound of the kernel's error: each layer's input kept to 2^-17, sums of 2 x 256
    products in FP32, SiLU to (4 + |z|) units of its value."""
    A, E = X.astype(np.float64), np.zeros(X.shape)
    for l, (w, c) in enumerate(zip(W, b)):
        aw = np.abs(w)
        keep = 2.0 ** -17 if 0 < l < len(W) - 1 else 0.0
        Z = A @ w + c
        E = (E + np.abs(A) * keep) @ aw + (2 * w.shape[0] + 2) * EPS * (np.abs(A) @ aw + np.abs(c))
        if l == len(W) - 1:
            return Z, 1.01 * E
        A = Z / (1.0 + np.exp(-Z))
        E = 1.1 * E + 2 * (4 + np.abs(Z)) * EPS * np.abs(A)          # |SiLU'| <= 1.1


@pytest.mark.parametrize("n", [1, 127, 128, 129, SMS * 128 - 1, SMS * 128 + 1, 3 * SMS * 128 + 77])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows(eng, n, shift):
    from sgl_analytic_gb300 import surrogate as S
    mlp = S.MLP(eng, width=256, depth=6, seed=11)
    rng = np.random.default_rng(n + shift)
    X = rng.uniform(-1.7, 1.7, (n, 8)).astype(np.float32)
    # shift: the rows start `shift` floats into an allocation
    (flat,) = S.to_device(eng, np.concatenate([np.zeros(shift, np.float32), X.ravel()]))
    Xd = flat[shift:].view(n, 8)
    Y = mlp.infer(Xd)
    mlp.stream.synchronize()
    W = [_bf16(w.cpu().numpy()) for w in mlp.W]
    b = [v.cpu().numpy().astype(np.float64) for v in mlp.b]
    rows = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n),
                                     rng.integers(0, n, 400)]))
    ref, bound = _exact_and_bound(W, b, X[rows])
    got = Y.cpu().numpy().astype(np.float64)
    assert got.shape == (n, 2)
    assert np.all(np.abs(got[rows] - ref) <= bound)


def test_large_preactivations_and_nan(eng):
    """Pre-activations far outside exp's range give 0 or z; a NaN stays in its row."""
    from sgl_analytic_gb300 import surrogate as S
    mlp = S.MLP(eng, width=256, depth=6, seed=3)
    rng = np.random.default_rng(0)
    X = rng.uniform(-1, 1, (260, 8)).astype(np.float32)
    X[3] *= 1e4
    X[130] = -1e4
    X[200, 5] = np.nan
    (Xd,) = S.to_device(eng, X)
    Y = mlp.infer(Xd)
    mlp.stream.synchronize()
    W = [_bf16(w.cpu().numpy()) for w in mlp.W]
    b = [v.cpu().numpy().astype(np.float64) for v in mlp.b]
    got = Y.cpu().numpy().astype(np.float64)
    with np.errstate(over="ignore", invalid="ignore"):
        ref, bound = _exact_and_bound(W, b, X)
    ok = np.arange(260) != 200
    assert np.all(np.isnan(got[200]))
    assert np.all(np.abs(got[ok] - ref[ok]) <= bound[ok])
