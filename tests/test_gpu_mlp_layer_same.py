"""sgl_mlp_layer and sgl_mlp_layer_grad give the numbers of the calls that they stand for: the GEMM on the split operands
with sgl_mlp_bias_act, and the GEMM with sgl_mlp_act_grad, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


def _engine(seed):
    import torch
    from sgl_analytic_gb300._lib import Engine
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch, Engine(0), lambda *s: torch.randn(s, generator=g, device="cuda")


@pytest.mark.parametrize("M,N,K", [(1, 2, 8), (127, 256, 8), (129, 255, 33), (300, 2, 256), (257, 256, 256), (700, 40, 17)])
@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("silu", [0, 1])
def test_layer(M, N, K, split, silu):
    torch, e, r = _engine(M + N + K)
    X, W, b = r(M, K), r(K, N), r(N)
    hi = X.bfloat16().float()
    A2, W2 = (torch.cat([hi, X - hi], 1), torch.cat([W, W], 0)) if split else (X, W)
    K2 = A2.shape[1]
    Z, Zr, Ar, Zb, A = (torch.zeros((M, N), device="cuda") for _ in range(5))
    torch.cuda.synchronize()
    e._check(e._L.sgl_gemm_bf16(e._h, M, N, K2, A2.data_ptr(), K2, 1, W2.data_ptr(), N, 1, Z.data_ptr(), N, 1, 1.0), "gemm")
    e._check(e._L.sgl_mlp_bias_act(e._h, M, N, Z.data_ptr(), b.data_ptr(), Zr.data_ptr(), Ar.data_ptr(), silu), "bias_act")
    e._check(e._L.sgl_mlp_layer(e._h, M, N, K, X.data_ptr(), W.data_ptr(), b.data_ptr(), Zb.data_ptr(), A.data_ptr(), silu,
                                split), "layer")
    torch.cuda.synchronize()
    assert torch.equal(Zb, Zr) and torch.equal(A, Ar)


@pytest.mark.parametrize("M,N,K", [(1, 8, 2), (127, 256, 2), (129, 255, 33), (257, 256, 256)])
def test_layer_gradient(M, N, K):
    torch, e, r = _engine(M + N + K)
    dZ, W, Zb = r(M, K), r(N, K), r(M, N)
    dA, ref, out = (torch.zeros((M, N), device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    e._check(e._L.sgl_gemm_bf16(e._h, M, N, K, dZ.data_ptr(), K, 1, W.data_ptr(), 1, K, dA.data_ptr(), N, 1, 1.0), "gemm")
    e._check(e._L.sgl_mlp_act_grad(e._h, M, N, dA.data_ptr(), Zb.data_ptr(), ref.data_ptr()), "act_grad")
    e._check(e._L.sgl_mlp_layer_grad(e._h, M, N, K, dZ.data_ptr(), W.data_ptr(), Zb.data_ptr(), out.data_ptr()), "layer_grad")
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
