"""Gauss instances split over parts of their cells, and batches whose buffers grow between graph replays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [2047, 2048, 4096 + 511, 65536])
@pytest.mark.parametrize("nk", [2, 64, 65, 129])
def test_split_instances_match_direct_sums(cells, nk):
    """Few k tiles and many cells: parts of whole tiles, the last one short, with a variance term; a second, small
    instance is not split.  FP64 within 1e-12 of the sum of magnitudes, mixed within 1e-6 (cfterm's bound)."""
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
    rng = np.random.default_rng(cells + nk)
    n = [cells, 5]
    kap, w = np.exp(rng.uniform(-5, 0, sum(n))), np.exp(rng.uniform(-4, 1, sum(n)))
    e = Engine(0)
    e.cfb_set(dict(inst_plane0=[0, 1, 2], plane_cells=[0, cells, cells + 5], kap=kap, w=w, nk=[nk, 2], dk=[0.37, 1.0],
                   closure=[0, 0], V=[0.3, 0.0], nstate=0, vp_D=np.zeros(2), vp_K=np.zeros(1), vp_w=np.zeros(1)))
    k = 0.37 * np.arange(nk)
    ph = np.outer(k, kap[:cells])
    c, s = -2 * np.sin(0.5 * ph) ** 2, np.where(ph < 0.3, -ph ** 3 / 6 * (1 - ph ** 2 / 20 * (1 - ph ** 2 / 42 * (1 - ph ** 2 / 72 * (
        1 - ph ** 2 / 110)))), np.sin(ph) - ph)
    ref = c @ w[:cells] - 0.15 * k * k + 1j * (s @ w[:cells])
    mag = np.abs(c) @ w[:cells] + 0.15 * k * k + np.abs(s) @ w[:cells]
    for precision, bar in ((SGL_FP64, 1e-12), (SGL_MIXED, 1e-6)):
        L = e.cfb_lnphi(precision)[:nk]
        assert L[0] == 0 and np.max(np.abs(L[1:] - ref[1:]) / mag[1:]) < bar


def test_template_cells_serve_both_precisions():
    """A template batch solved in one precision, then the other: each finds its cells."""
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
    rng = np.random.default_rng(1)
    F, g = rng.uniform(0.1, 1, (8, 40)), rng.uniform(0.1, 1, 40)
    u, v = rng.uniform(0.1, 1, (3, 8)), rng.uniform(0.1, 1, (3, 8))
    out = {}
    for first in (SGL_MIXED, SGL_FP64):
        e = Engine(0)
        e.cfb_set_separable(F, g, [0, 2, 3], [33, 70], [0.2, 0.1], [0.0, 0.1], u, v)
        for p in (first, SGL_MIXED, SGL_FP64):
            out[first, p] = e.cfb_lnphi(p)
    assert np.array_equal(out[SGL_MIXED, SGL_MIXED], out[SGL_FP64, SGL_MIXED])
    assert np.array_equal(out[SGL_MIXED, SGL_FP64], out[SGL_FP64, SGL_FP64])
    assert np.max(np.abs(out[SGL_MIXED, SGL_MIXED] - out[SGL_MIXED, SGL_FP64])) < 1e-5 * np.max(np.abs(out[SGL_MIXED, SGL_FP64]))


def test_graph_survives_the_other_precision():
    """A captured mixed step replayed after FP64 and wider calls on the same batch."""
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
    from sgl_analytic_gb300.cfbatch import make_batch
    b = make_batch(4, seed=3, nm=4, nb=4, nk_range=(256, 512), nk_step=1, max_planes=3)
    e = Engine(0)
    e.cfb_set(b.arrays())
    x, wide = np.linspace(-0.4, 1.5, 100), np.linspace(-0.4, 1.5, 3000)
    a, _ = e.cfb_pdf(x, SGL_MIXED)
    e.cfb_pdf(wide, SGL_FP64)
    c, _ = e.cfb_pdf(x, SGL_MIXED)
    assert np.array_equal(a, c)
