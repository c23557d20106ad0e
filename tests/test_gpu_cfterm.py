"""The packed FP32 compensated terms (cfterm.cuh) of the 1-D sweep and of the batched solver against FP64, at the
edges of their groups (8 cells) and tiles (512 cells) and over phases from 1e-6 to 2.5e7.

Bound: a term's parts carry the rounding of r (1.5 ulp), of a degree-6 Horner chain (3 ulp) and of the weight, and
4 FMAs of a lane's group, each at most 2^-24 of the running group sum: 10 x 2^-24 = 6e-7 of the sum of the terms'
magnitudes; 1e-6 is asserted, for the real and the imaginary part separately."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = 1e-6


def _reference(kk, kap, w):
    ph = np.outer(kk, kap)
    c = -2 * np.sin(0.5 * ph) ** 2
    p2 = ph * ph
    s = np.where(np.abs(ph) < 0.3, -ph * p2 / 6 * (1 - p2 / 20 * (1 - p2 / 42 * (1 - p2 / 72 * (1 - p2 / 110)))), np.sin(ph) - ph)
    return c @ w, s @ w, np.abs(c) @ np.abs(w), np.abs(s) @ np.abs(w)


@pytest.mark.parametrize("nc", [1, 7, 8, 9, 504, 511, 512, 513, 2049])
@pytest.mark.parametrize("nk,lo,hi", [(1, 1.0, 1.0), (17, 1e-6, 1e-2), (257, 1e-2, 1e2), (300, 1e2, 2.5e7)])
def test_sweep_terms(nc, nk, lo, hi):
    from sgl_analytic_gb300._lib import SGL_MIXED, Engine
    rng = np.random.default_rng(nc * 1000 + nk)
    kap = rng.choice([-1.0, 1.0], nc) * np.exp(rng.uniform(np.log(0.05), 0.0, nc))
    w = np.exp(rng.uniform(-8, 2, nc))
    kk = np.geomspace(lo, hi, nk)
    e = Engine(0)
    e.sweep_set_cells(kap, w)
    out = e.sweep(kk, SGL_MIXED)
    re, im, are, aim = _reference(kk, kap, w)
    assert np.max(np.abs(out.real - re) / are) < BOUND
    assert np.max(np.abs(out.imag - im) / aim) < BOUND


def test_zero_kappa_and_zero_k_give_zero():
    from sgl_analytic_gb300._lib import SGL_MIXED, Engine
    e = Engine(0)
    e.sweep_set_cells(np.array([0.0, 0.3, 0.0]), np.array([1.0, 0.0, 2.0]))
    assert np.all(e.sweep(np.array([0.0, 1.0, 1e6]), SGL_MIXED) == 0)


@pytest.mark.parametrize("cells", [[1], [7, 1, 9], [512, 513, 3]])
@pytest.mark.parametrize("nk", [2, 63, 65, 257])
def test_batch_terms(cells, nk):
    """The same through sgl_cfb_lnphi: ragged planes, k grids around the tile widths."""
    from sgl_analytic_gb300._lib import SGL_MIXED, Engine
    rng = np.random.default_rng(sum(cells) + nk)
    nc = sum(cells)
    kap, w = np.exp(rng.uniform(-5, 0, nc)), np.exp(rng.uniform(-4, 1, nc))
    e = Engine(0)
    e.cfb_set(dict(inst_plane0=[0, len(cells)], plane_cells=np.concatenate([[0], np.cumsum(cells)]), kap=kap, w=w, nk=[nk],
                   dk=[0.37], closure=[0], V=[0.0], nstate=0, vp_D=np.zeros(1), vp_K=np.zeros(1), vp_w=np.zeros(1)))
    out = e.cfb_lnphi(SGL_MIXED)
    re, im, are, aim = _reference(0.37 * np.arange(1, nk), kap, w)
    assert out[0] == 0
    assert np.max(np.abs(out.real[1:] - re) / are) < BOUND
    assert np.max(np.abs(out.imag[1:] - im) / aim) < BOUND
