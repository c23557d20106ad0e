"""The fused xi kernel harmonic by harmonic, against the FP64 path: one group at a time and no residual row element, so that
each harmonic's squares are the whole signal.

Bound: T's FP32 sums, E, and their three TF32 products are each good to 2^-20 of the sums' random magnitude, which is that of
the sums themselves; squaring doubles it: 6 x 2^-20 = 6e-6 of the largest value, 1e-5 is asserted."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [0, 1, 2])
@pytest.mark.parametrize("rows,cells,nk,nkg", [(1, 1, 101, 101), (3, 4, 101, 7), (4, 5, 128, 8), (5, 15, 41, 9),
                                               (32, 17, 101, 17), (36, 49, 101, 101), (47, 192, 127, 23),
                                               (48, 200, 101, 101), (49, 33, 101, 101), (97, 64, 65, 30)])
def test_one_harmonic(m, rows, cells, nk, nkg):
    from sgl_analytic_gb300 import Lam, Population
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED
    pop = Population.load(GOLDEN / "pop_zs1_sub.npz")
    rng = np.random.default_rng(1000 * rows + 10 * cells + m)
    n_k, n_g = pop.ce_k.size - 1, pop.ce_g.size - 1
    idx = []
    for c, ik in enumerate(np.sort(rng.choice(n_k, cells, replace=False))):
        n = n_g if c == 0 else int(rng.integers(1, 31))
        idx.append(ik * n_g + np.sort(rng.choice(n_g, n, replace=False)))
    idx = np.concatenate(idx).astype(np.int32)
    r = rng.standard_normal((rows, idx.size + 1)) * 1e-2
    r[:, -1] = 0.0
    pop.xg_m, pop.xg_nrow, pop.xg_nidx = np.array([m], np.int32), np.array([rows], np.int32), np.array([idx.size], np.int32)
    pop.xg_idx, pop.xg_rows = idx, r.ravel()
    lam = Lam(pop, xi=True, xi_prune=0.0)
    kk, kg = np.linspace(0.0, 900.0, nk), np.linspace(0.0, 700.0, nkg)
    q64, qmx = (lam.engine.xi_term(kk, kg, p) for p in (SGL_FP64, SGL_MIXED))
    assert np.max(np.abs(q64)) > 0
    assert np.max(np.abs(qmx - q64)) <= 1e-5 * np.max(np.abs(q64))
