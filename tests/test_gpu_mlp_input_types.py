"""MLP.forward on inputs that are not packed float32: values that every type holds give the float32 result."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float16", "bfloat16", "int32", "int64", "float64"])
@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("n", [1, 129, 600])
def test_forward_converts_its_input(dtype, split, n):
    import torch
    from sgl_analytic_gb300._lib import Engine
    from sgl_analytic_gb300.surrogate import MLP
    m = MLP(Engine(0), width=64, depth=2, seed=3, split=split)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    Xi = torch.randint(-3, 4, (n, 8), device="cuda", generator=g)
    X, Xf = Xi.to(getattr(torch, dtype)), Xi.to(torch.float32)
    torch.cuda.synchronize()                      # torch's stream is not ordered with the engine's
    a, b = m.forward(X, keep=True), m.forward(Xf)
    m.stream.synchronize()
    assert m._acts[0].dtype == torch.float32
    assert torch.equal(a, b)
