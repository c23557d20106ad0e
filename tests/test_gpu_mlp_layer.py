"""sgl_mlp_layer, sgl_gemm_bf16 with a long K and the column sums at the edges of their tiles, against the same
arithmetic in torch FP64 on the same BF16-rounded operands.

Bounds: products of BF16 values are exact in FP32 and accumulate over K terms in FP32 (2^-23 each, truncation
included): 2^-23 sqrt(K) of the sum of magnitudes is typical, K 2^-23 the worst; 32 x 2^-23 = 4e-6 of it is asserted (sums stay below it on these inputs' random signs).
Column sums are FP64 sums rounded to FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(seed):
    import torch
    from sgl_analytic_gb300._lib import Engine
    e = Engine(0)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch, e, lambda *s: torch.randn(s, generator=g, device="cuda")


def _bf(x):
    return x.bfloat16().double()


@pytest.mark.parametrize("M,N,K", [(1, 2, 8), (127, 256, 8), (129, 255, 33), (300, 2, 256), (257, 256, 256)])
@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("silu", [0, 1])
def test_layer(M, N, K, split, silu):
    torch, e, r = _setup(M + N + K)
    X, W, b = r(M, K), r(K, N), r(N)
    Zb, A = torch.zeros((M, N), device="cuda"), torch.zeros((M, N), device="cuda")
    torch.cuda.synchronize()
    e._check(e._L.sgl_mlp_layer(e._h, M, N, K, X.data_ptr(), W.data_ptr(), b.data_ptr(), Zb.data_ptr(), A.data_ptr(), silu,
                                split), "layer")
    torch.cuda.synchronize()
    Xe = _bf(X) + (_bf(X - X.bfloat16().float()) if split else 0)
    z = Xe @ _bf(W) + b.double()
    mag = Xe.abs() @ _bf(W).abs() + b.double().abs()
    assert float(((Zb.double() - z).abs() / mag).max()) < 4e-6
    a = z * torch.sigmoid(z) if silu else z
    assert float(((A.double() - a).abs() / mag).max()) < 4e-6


@pytest.mark.parametrize("M,N,K", [(1, 8, 2), (127, 256, 2), (129, 255, 33), (257, 256, 256)])
def test_layer_gradient(M, N, K):
    torch, e, r = _setup(M + N + K)
    dZ, W, Zb = r(M, K), r(N, K), r(M, N)
    out = torch.zeros((M, N), device="cuda")
    torch.cuda.synchronize()
    e._check(e._L.sgl_mlp_layer_grad(e._h, M, N, K, dZ.data_ptr(), W.data_ptr(), Zb.data_ptr(), out.data_ptr()), "grad")
    torch.cuda.synchronize()
    s = torch.sigmoid(Zb.double())
    f = s * (1 + Zb.double() * (1 - s))
    mag = _bf(dZ).abs() @ _bf(W).abs().T
    assert float(((out.double() - (_bf(dZ) @ _bf(W).T) * f).abs() / mag).max()) < 4e-6


@pytest.mark.parametrize("M,N,K", [(256, 256, 8191), (256, 256, 8192), (8, 256, 16384), (256, 2, 12301), (130, 300, 9000)])
def test_weight_gradient(M, N, K):
    torch, e, r = _setup(K)
    A, B = r(K, M), r(K, N)
    C = torch.zeros((M, N), device="cuda")
    torch.cuda.synchronize()
    e._check(e._L.sgl_gemm_bf16(e._h, M, N, K, A.data_ptr(), 1, M, B.data_ptr(), N, 1, C.data_ptr(), N, 1, 0.5), "gemm")
    torch.cuda.synchronize()
    ref, mag = 0.5 * _bf(A).T @ _bf(B), 0.5 * _bf(A).abs().T @ _bf(B).abs()
    assert float(((C.double() - ref).abs() / mag).max()) < 4e-6


@pytest.mark.parametrize("M,N", [(0, 3), (1, 1), (63, 127), (64, 128), (65, 129), (16384, 256)])
def test_column_sums(M, N):
    torch, e, r = _setup(M + N)
    X, out = r(max(M, 1), N), torch.ones(N, device="cuda")
    torch.cuda.synchronize()
    e._check(e._L.sgl_mlp_col_sum(e._h, M, N, X.data_ptr(), out.data_ptr()), "col_sum")
    torch.cuda.synchronize()
    ref = X[:M].double().sum(0)
    assert float((out.double() - ref).abs().max()) <= 2.0 ** -23 * float(ref.abs().max() + 1e-30)


def test_forward_takes_a_strided_input():
    import torch
    from sgl_analytic_gb300._lib import Engine
    from sgl_analytic_gb300.surrogate import MLP
    m = MLP(Engine(0), seed=3)
    X = torch.rand((600, 16), device="cuda")
    Xc = X[:, ::2].contiguous()
    torch.cuda.synchronize()                      # torch's stream is not ordered with the engine's
    strided, plain = m.forward(X[:, ::2]), m.forward(Xc)
    m.stream.synchronize()
    assert torch.equal(strided.cpu(), plain.cpu())
