"""The sliced FP64 GEMM (oz_gemm.cu) where its sizes are awkward, through the entry points that use it.

Bounds: the separable ln Phi within 1e-10 of the dense direct sum (the bar of the FP64 path), and the inversion of a
given Phi within 1e-12 of its largest value of the same sums in extended precision: the transforms' terms are at most
|Phi| dk^2 k times 2^-53 each."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nkg", [(75, 2687), (127, 2001), (129, 1603), (301, 1001), (6001, 64)])
def test_separable_grids_match_direct_sums(nk, nkg):
    """Rows, columns and K off every tile size; the last grid has more rows than one batch of digits holds."""
    from oracle.lam_oracle import psi1_direct
    from sgl_analytic_gb300 import Lam, Population
    pop = Population.load(GOLDEN / "pop_zs1_sub.npz")
    kk = np.linspace(0.0, 1010.4632803971984, nk)
    kg = np.linspace(0.0, 808.3706243177588, nkg)
    L = Lam(pop, xi=False)(kk, kg)
    i, j = np.unique(np.linspace(0, nk - 1, 7).astype(int)), np.unique(np.linspace(0, nkg - 1, 9).astype(int))
    ref = psi1_direct(pop.k0, pop.g0, pop.w0, kk[i], kg[j])
    d = np.abs(L[np.ix_(i, j)] - ref)
    assert np.all(d <= np.where(np.abs(ref) > 100, 1e-12 * np.abs(ref), 1e-10)), d.max()


def _grid(nk, ng, nkap, ngam):
    return dict(nk_k=nk, nk_g=ng, n_kap=nkap, n_gam=ngam, k_k_max=120.0, k_g_max=110.0, kap_min=-0.3, kap_max=0.99,
                gam_max=0.8, sigma=0.05, phi_at_k_cut=1e-9, phi_at_g_cut=1e-9)


@pytest.mark.parametrize("nk,ng,nkap,ngam", [(331, 1203, 601, 257), (512, 640, 513, 320)])
def test_inversion_of_a_given_phi(nk, ng, nkap, ngam):
    """The Hankel and kappa transforms on odd and on full tiles: a Phi that spans eight decades, against NumPy."""
    from oracle.invert_oracle import em_correction, p_vector_joint, path_integral
    from sgl_analytic_gb300._lib import SGL_FP64, Engine
    g = _grid(nk, ng, nkap, ngam)
    kk, kg = np.linspace(0, g["k_k_max"], nk), np.linspace(0, g["k_g_max"], ng)
    phi = np.exp(-0.5 * (0.05 * kk[:, None]) ** 2 - 0.5 * (0.05 * kg[None, :]) ** 2 - 0.01j * kk[:, None])
    x = np.linspace(-0.2, 0.4, 101)
    P, m = Engine(0).invert_phi(phi, g, x, precision=SGL_FP64)
    kap, gam = np.linspace(g["kap_min"], g["kap_max"], nkap), np.linspace(0, g["gam_max"], ngam)
    P3 = p_vector_joint(kk, kg, phi, kap, gam)
    a, b = em_correction(kk, kg, phi[:, 0], phi[:, 1], kap, gam)
    P3 = P3 + a[:, None] + b[:, None] * gam[None, :] ** 2
    ref = path_integral(P3, kap, gam, x, g["gam_max"], min(6 * g["sigma"], g["gam_max"]))
    P = P * m["norm"]
    assert np.max(np.abs(P - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_nan_in_phi_is_reported():
    from sgl_analytic_gb300._lib import SGL_FP64, Engine
    g = _grid(512, 640, 513, 320)
    phi = np.ones((512, 640), complex)
    phi[200, 300] = np.nan
    with pytest.raises(RuntimeError):
        Engine(0).invert_phi(phi, g, np.linspace(-0.2, 0.4, 11), precision=SGL_FP64)


@pytest.mark.parametrize("nk", [63, 64, 65, 160])
@pytest.mark.parametrize("spacing", ["uniform", "offset", "geometric"])
def test_fp64_sweep_rows(nk, spacing):
    """The FP64 separable sweep on uniform rows (the split half angles from 64 rows on, a last warp partly filled),
    on uniform rows that do not start at 0 and on rows of no common step, against the dense sum."""
    from oracle.lam_oracle import psi1_direct
    from sgl_analytic_gb300 import Lam, Population
    pop = Population.load(GOLDEN / "pop_zs1_sub.npz")
    kk = {"uniform": np.linspace(0.0, 900.0, nk), "offset": np.linspace(3.7, 411.3, nk),
          "geometric": np.geomspace(1e-4, 900.0, nk)}[spacing]
    kg = np.linspace(0.0, 700.0, 200000 // nk + 1)
    L = Lam(pop, xi=False)(kk, kg)
    i, j = np.unique([0, 1, 31, 32, 33, nk - 2, nk - 1]), np.array([0, 1, 500, kg.size - 1])
    ref = psi1_direct(pop.k0, pop.g0, pop.w0, kk[i], kg[j])
    d = np.abs(L[np.ix_(i, j)] - ref)
    assert np.all(d <= np.where(np.abs(ref) > 100, 1e-12 * np.abs(ref), 1e-10)), d.max()


def test_subnormal_products():
    """A Phi scaled by 2^-1015 takes the smaller outputs below the normal numbers: P and norm scale with it.  Subnormal
    steps of 2^-1074 in a few hundred terms stay below 1e-12 of the largest sums (above 2^-1015)."""
    from sgl_analytic_gb300._lib import SGL_FP64, Engine
    g = _grid(331, 1203, 601, 257)
    kk, kg = np.linspace(0, g["k_k_max"], g["nk_k"]), np.linspace(0, g["k_g_max"], g["nk_g"])
    phi = np.exp(-0.5 * (0.05 * kk[:, None]) ** 2 - 0.5 * (0.05 * kg[None, :]) ** 2 - 0.01j * kk[:, None])
    x = np.linspace(-0.2, 0.4, 101)
    e = Engine(0)
    P, m = e.invert_phi(phi, g, x, precision=SGL_FP64)
    Q, n = e.invert_phi(phi * 2.0 ** -1015, g, x, precision=SGL_FP64)
    assert abs(n["norm"] * 2.0 ** 1015 - m["norm"]) <= 1e-12 * abs(m["norm"])
    assert np.max(np.abs(Q - P)) <= 2e-12 * np.max(np.abs(P))
