"""The mixed vp chain where a shell's z spreads over more than FP32's range: states that are negligible after one shell and
the largest after the next.  k kappa are multiples of pi, so that every cell sum is a small dyadic number, exact in FP32,
and no sum of states cancels; rates of a closure add up to 0.  What is left is the chain: some 2^12 operations of 2^-48
each, 1e-10 (1 + |ln R|) against the FP64 path.  Where that path's own range ends (squares of the states below 1e-308)
both refuse."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _closure(rates, weight, mix):
    """One linear group per shell (D = rate u), all on one cell at kappa = 1, gamma = 0; transitions mix per shell towards
    the stationary weights (0: none)."""
    g = np.load(GOLDEN / "vp_zs1_sub.npz")
    u, w, n = g["u"], g["w"], len(rates)
    K = (1 - mix) * np.eye(48) + mix * np.broadcast_to(w, (48, 48))
    return dict(u=u, w=w, K=np.repeat(K[None], n - 1, 0), shear_var=np.float64(0.0), ku=np.ones(1), gu=np.zeros(1),
                cu=np.zeros(n, np.int32), cw=np.full(n, weight), gstart=np.arange(n + 1, dtype=np.int64),
                sh_g=np.arange(n + 1, dtype=np.int32), ga=np.array(rates, float), gb=np.zeros(n), gc=np.zeros(n),
                glo=np.zeros(n, np.int32), ghi=np.full(n, 47, np.int32))


@pytest.mark.parametrize("weight", [0.5, 2.0, 4.0, 12.0])
@pytest.mark.parametrize("mix", [0.0, 1e-6, 0.3])
@pytest.mark.parametrize("rates", [(1.0, -1.0), (1.0, 0.5, -2.0, 0.25, 0.25), (1.0, 1.0, 1.0, -1.5, -1.5)])
@pytest.mark.parametrize("shape", [(33, 40), (40, 20)])
def test_states_that_come_back(weight, mix, rates, shape):
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
    e = Engine(0)
    e.set_vp(_closure(rates, weight, mix))
    k, q = np.pi * np.arange(shape[0]), np.linspace(0.0, 5.0, shape[1])               # Re z = 0 or -2 weight rate u
    try:
        a = e.vp_lnR(k, q, SGL_FP64)
    except RuntimeError:
        with pytest.raises(RuntimeError):
            e.vp_lnR(k, q, SGL_MIXED)
        return
    b = e.vp_lnR(k, q, SGL_MIXED)
    assert np.all(np.abs(a - b) <= 1e-10 * (1 + np.abs(a)))
    if mix == 0.0:
        assert np.max(np.abs(a)) < 1e-12 * (1 + 30 * weight)                          # the shells cancel
