"""Which FP64 GEMMs run sliced: enough work, and tiles and K that fill the chip.  Long K on few tiles stays on the SIMT
kernel's K slices; either way the transforms meet the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,ng,nkap,ngam,route", [(64, 60000, 64, 64, "f64"), (128, 16000, 128, 64, "f64"),
                                                   (30, 8000, 100, 500, "f64"), (60, 4000, 100, 500, "oz"),
                                                   (200, 1000, 200, 500, "oz"), (100, 500, 100, 200, "f64")])
def test_hankel_route(nk, ng, nkap, ngam, route):
    from oracle.invert_oracle import em_correction, p_vector_joint, path_integral
    from sgl_analytic_gb300._lib import SGL_FP64, Engine
    g = dict(nk_k=nk, nk_g=ng, n_kap=nkap, n_gam=ngam, k_k_max=60.0, k_g_max=110.0, kap_min=-0.3, kap_max=0.99, gam_max=0.8,
             sigma=0.05, phi_at_k_cut=1e-9, phi_at_g_cut=1e-9)
    kk, kg = np.linspace(0, g["k_k_max"], nk), np.linspace(0, g["k_g_max"], ng)
    phi = np.exp(-0.5 * (0.05 * kk[:, None]) ** 2 - 0.5 * (0.05 * kg[None, :]) ** 2 - 0.01j * kk[:, None])
    x = np.linspace(-0.2, 0.4, 101)
    e = Engine(0)
    e.profile(True)
    e.stats(reset=True)
    P, m = e.invert_phi(phi, g, x, precision=SGL_FP64)
    names = set(e.stats())
    assert f"gemm_{route}_hankel" in names and f"gemm_{'oz' if route == 'f64' else 'f64'}_hankel" not in names
    kap, gam = np.linspace(g["kap_min"], g["kap_max"], nkap), np.linspace(0, g["gam_max"], ngam)
    a, b = em_correction(kk, kg, phi[:, 0], phi[:, 1], kap, gam)
    P3 = p_vector_joint(kk, kg, phi, kap, gam) + a[:, None] + b[:, None] * gam[None, :] ** 2
    ref = path_integral(P3, kap, gam, x, g["gam_max"], min(6 * g["sigma"], g["gam_max"]))
    assert np.max(np.abs(P * m["norm"] - ref)) <= 1e-12 * np.max(np.abs(ref))
