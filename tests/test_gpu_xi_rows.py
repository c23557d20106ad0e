"""The fused xi kernel at the edges of its tiles: row counts around its row quads and its 48-row limit, kappa cells of 1
to 110 entries, and numbers of kappa cells around its K blocks and its twelve producers' turns, against the FP64 path.

Bound of a row's sums: operands to 2^-21 twice and FP32 sums of its entries and cells on terms of at most 2 |row|."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _groups(rng, rows, cells, n_k, n_g):
    """One group per harmonic: `cells` kappa cells, the first of them full, the others of 1 to 30 entries."""
    out = []
    for m in (0, 1, 2):
        idx = []
        for c, ik in enumerate(np.sort(rng.choice(n_k, cells, replace=False))):
            n = n_g if c == 0 else int(rng.integers(1, 31))
            idx.append(ik * n_g + np.sort(rng.choice(n_g, n, replace=False)))
        idx = np.concatenate(idx).astype(np.int32)
        out.append((m, idx, rng.standard_normal((rows, idx.size + 1)) * np.exp(rng.uniform(-3, 0, (rows, 1))) * 1e-2))
    return out


@pytest.mark.parametrize("rows,cells,nk,nkg", [(1, 1, 101, 101), (3, 4, 101, 7), (4, 5, 128, 8), (5, 15, 1 + 40, 9),
                                               (31, 16, 101, 101), (32, 17, 101, 17), (33, 48, 100, 33), (36, 49, 101, 101),
                                               (41, 97, 101, 50), (47, 192, 127, 23), (48, 200, 101, 101), (49, 33, 101, 101),
                                               (97, 64, 65, 30)])
def test_mixed_against_fp64(rows, cells, nk, nkg):
    from sgl_analytic_gb300 import Lam, Population
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED
    pop = Population.load(GOLDEN / "pop_zs1_sub.npz")
    rng = np.random.default_rng(rows * 1000 + cells)
    n_k, n_g = pop.ce_k.size - 1, pop.ce_g.size - 1
    gr = _groups(rng, rows, cells, n_k, n_g)
    pop.xg_m = np.array([g[0] for g in gr], np.int32)
    pop.xg_nrow = np.array([rows] * 3, np.int32)
    pop.xg_nidx = np.array([g[1].size for g in gr], np.int32)
    pop.xg_idx = np.concatenate([g[1] for g in gr])
    pop.xg_rows = np.concatenate([g[2].ravel() for g in gr])
    lam = Lam(pop, xi=True, xi_prune=0.0)
    kk, kg = np.linspace(0.0, 900.0, nk), np.linspace(0.0, 700.0, nkg)
    q64, qmx = (lam.engine.xi_term(kk, kg, p) for p in (SGL_FP64, SGL_MIXED))
    bound = 0.0
    for m, idx, row in gr:
        S = np.abs(row[:, :-1]).sum(1) + 1000.0 * np.abs(row[:, -1])
        delta = 2 * S * (2.0 ** -20 + (cells + 110 + 16) * 2.0 ** -24)
        bound += np.sum(2 * 2 * (2 * S) * delta)
    assert np.max(np.abs(qmx - q64)) <= bound
