"""Column sums on both sides of the row count from which they take two passes; FP64 sums rounded to FP32."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [0, 1, 255, 32767, 32768, 32769, 100003])
@pytest.mark.parametrize("N", [1, 8, 129])
def test_column_sums(M, N):
    import torch
    from sgl_analytic_gb300._lib import Engine
    e = Engine(0)
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    X, out = torch.randn((max(M, 1), N), device="cuda", generator=g), torch.ones(N, device="cuda")
    torch.cuda.synchronize()
    e._check(e._L.sgl_mlp_col_sum(e._h, M, N, X.data_ptr(), out.data_ptr()), "col_sum")
    torch.cuda.synchronize()
    ref = X[:M].double().sum(0)
    assert torch.all((out.double() - ref).abs() <= 2.0 ** -24 * ref.abs() + 1e-12)
