"""The FP64 xi groups' products in one launch on grids too small for the slices, the leading rows apart from them on larger
ones: the same values at the points that both grids have."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nkg", [(1, 1), (7, 9), (33, 40), (128, 5)])
def test_small_grids_take_one_launch(nk, nkg):
    from sgl_analytic_gb300 import Lam, Population
    from sgl_analytic_gb300._lib import SGL_FP64
    lam = Lam(Population.load(GOLDEN / "pop_zs1_sub.npz"), xi=True)
    e = lam.engine
    kk, kg = np.linspace(0.0, 900.0, 128), np.linspace(0.0, 700.0, 101)
    i, j = np.unique(np.linspace(0, 127, nk).astype(int)), np.unique(np.linspace(0, 100, nkg).astype(int))
    big = e.xi_term(kk, kg, SGL_FP64)[np.ix_(i, j)]
    e.profile(True)
    e.stats(reset=True)
    small = e.xi_term(kk[i], kg[j], SGL_FP64)
    assert "gemm_f64_xi_lead" not in e.stats() and "gemm_oz_xi" not in e.stats()
    assert np.all(np.abs(small - big) <= 1e-14 + 1e-10 * np.abs(big))
