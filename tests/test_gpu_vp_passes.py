"""A line of points whose states do not fit one pass (8 GiB: 18,101 shells and 608 points take two): each pass has its own
rows."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


def test_a_line_in_two_passes():
    """One cell per shell, linear rates.  The line in two passes gives the bits of its halves, which take one each."""
    from sgl_analytic_gb300._lib import SGL_MIXED, Engine
    g = np.load(GOLDEN / "vp_zs1_sub.npz")
    n, rng = 18101, np.random.default_rng(2)
    e = Engine(0)
    e.set_vp(dict(u=g["u"], w=g["w"], K=np.broadcast_to(g["K"][0], (n - 1, 48, 48)), shear_var=np.float64(0.0),
                  ku=np.linspace(0.01, 1.0, 64), gu=np.linspace(0.0, 0.5, 64), cu=rng.integers(0, 64, n).astype(np.int32),
                  cw=rng.uniform(1e-4, 1e-3, n), gstart=np.arange(n + 1, dtype=np.int64),
                  sh_g=np.arange(n + 1, dtype=np.int32), ga=rng.uniform(0.5, 1.0, n), gb=np.zeros(n), gc=np.zeros(n),
                  glo=np.zeros(n, np.int32), ghi=np.full(n, 47, np.int32)))
    k, q = np.linspace(0.0, 200.0, 608), np.full(1, 3.0)
    whole = e.vp_lnR(k, q, SGL_MIXED)
    halves = np.concatenate([e.vp_lnR(k[:304], q, SGL_MIXED), e.vp_lnR(k[304:], q, SGL_MIXED)])
    assert np.array_equal(whole, halves)
    assert np.unique(whole[:, 0]).size == 608
