"""The sliced FP64 GEMM's scales where a column of its left operand is empty or not finite: Phi is the Hankel transform's
left operand, with k_gamma as the product's inner index."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu

GRID = dict(nk_k=331, nk_g=1203, n_kap=601, n_gam=257, k_k_max=120.0, k_g_max=110.0, kap_min=-0.3, kap_max=0.99,
            gam_max=0.8, sigma=0.05, phi_at_k_cut=1e-9, phi_at_g_cut=1e-9)
X = np.linspace(-0.2, 0.4, 101)


def _phi():
    kk, kg = np.linspace(0, GRID["k_k_max"], GRID["nk_k"]), np.linspace(0, GRID["k_g_max"], GRID["nk_g"])
    return kk, kg, np.exp(-0.5 * (0.05 * kk[:, None]) ** 2 - 0.5 * (0.05 * kg[None, :]) ** 2 - 0.01j * kk[:, None])


def _oracle(kk, kg, phi):
    from oracle.invert_oracle import em_correction, p_vector_joint, path_integral
    kap, gam = np.linspace(GRID["kap_min"], GRID["kap_max"], GRID["n_kap"]), np.linspace(0, GRID["gam_max"], GRID["n_gam"])
    a, b = em_correction(kk, kg, phi[:, 0], phi[:, 1], kap, gam)
    P3 = p_vector_joint(kk, kg, phi, kap, gam) + a[:, None] + b[:, None] * gam[None, :] ** 2
    return path_integral(P3, kap, gam, X, GRID["gam_max"], min(6 * GRID["sigma"], GRID["gam_max"]))


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40, 2.0 ** -900])
@pytest.mark.parametrize("empty", [[700], [5, 6, 7, 640, 1202], list(range(900, 1203))])
def test_empty_columns_beside_small_ones(scale, empty):
    """k_gamma columns of zeros in a Phi of any magnitude.  The transforms' terms are at most |Phi| dk^2 k times 2^-53 each:
    1e-12 of the largest value, as for a Phi without empty columns."""
    from sgl_analytic_gb300._lib import SGL_FP64, Engine
    kk, kg, phi = _phi()
    phi[:, empty] = 0.0
    P, m = Engine(0).invert_phi(phi * scale, GRID, X, precision=SGL_FP64)
    ref = _oracle(kk, kg, phi)
    assert np.max(np.abs(P * (m["norm"] / scale) - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_an_infinity_stays_one():
    """An infinite row element of the xi groups: infinities and NaN where FP64 products have them, as the same rows of a
    grid too small for the slices (below 0.4 GFLOP) show."""
    from sgl_analytic_gb300 import Lam, Population
    from sgl_analytic_gb300._lib import SGL_FP64
    pop = Population.load(GOLDEN / "pop_zs1_sub.npz")
    rng = np.random.default_rng(5)
    n_k, n_g = pop.ce_k.size - 1, pop.ce_g.size - 1
    idx = np.concatenate([ik * n_g + np.sort(rng.choice(n_g, 12, replace=False)) for ik in range(330)]).astype(np.int32)
    rows = rng.standard_normal((36, idx.size + 1)) * 1e-2
    rows[7, 40] = np.inf
    pop.xg_m, pop.xg_nrow, pop.xg_nidx = np.array([1], np.int32), np.array([36], np.int32), np.array([idx.size], np.int32)
    pop.xg_idx, pop.xg_rows = idx, rows.ravel()
    lam = Lam(pop, xi=True, xi_prune=0.0)
    kk, kg = np.linspace(0.0, 900.0, 101), np.linspace(0.0, 700.0, 101)          # 0.48 GFLOP
    sel = np.array([0, 1, 50, 100])
    q, few = lam.engine.xi_term(kk, kg, SGL_FP64), lam.engine.xi_term(kk[sel], kg, SGL_FP64)
    assert np.isinf(few.imag).any()
    for a, b in ((q.real[sel], few.real), (q.imag[sel], few.imag)):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.array_equal(a[np.isinf(a)], b[np.isinf(b)])
