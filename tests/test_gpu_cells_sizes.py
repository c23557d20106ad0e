"""The xi_lin deposit at the edges of its work items (4096 points, 16 radii a batch, 32 lanes), against the oracle:
the bars of test_gpu_cells.py."""
import numpy as np
import pytest

from tests import cells_replay as CR

pytestmark = pytest.mark.gpu


def _object(rng, n, n_radii, tang):
    """n points on n_radii distinct radii from 1e-4 to 30 Mpc, some outside the coarse box."""
    K = rng.choice([-1.0, 1.0], n) * np.exp(rng.uniform(np.log(1e-8), np.log(40.0), n))
    return dict(K=K, G=np.exp(rng.uniform(np.log(1e-10), np.log(40.0), n)), W=np.exp(rng.uniform(-5, 2, n)),
                R=rng.choice(np.geomspace(1e-4, 30.0, n_radii), n), shell=0, beta=float(rng.uniform(0.5, 3)), tang=tang)


@pytest.mark.parametrize("sizes,n_radii", [([1], 1), ([31, 32, 33], 5), ([512, 513], 16), ([4095, 4096, 4097], 17),
                                           ([8200, 3], 4000), ([300, 40], 1)])
@pytest.mark.parametrize("pos", [False, True])
def test_items_match_oracle(sizes, n_radii, pos):
    from oracle.cells_oracle import CellsOracle
    from sgl_analytic_gb300.cells import Cells
    rng = np.random.default_rng(sum(sizes) + n_radii)
    d = CR.load()
    xi = dict(kp=d["xi_kp"], c=d["xi_c"], mmax=2, pos=pos)
    objs = [_object(rng, n, n_radii, i % 3 != 2) for i, n in enumerate(sizes)]
    c, o = Cells(1, 1, xi=xi), CellsOracle(1, 1, xi=xi)
    for a in (c, o):
        a.xi_begin(35.0)
    c.add_many(objs)
    for ob in objs:
        o.add(ob["K"], ob["G"], ob["W"], 0, ob["beta"], R=ob["R"], tang=ob["tang"])
    for a in (c, o):
        a.xi_end(0)
    np.testing.assert_allclose(np.asarray(c.H0), np.asarray(o.H0), rtol=1e-12)
    assert len(c.xi_groups) == len(o.xi_groups)
    for g, h in zip(c.xi_groups, o.xi_groups):
        assert g["m"] == h["m"] and np.array_equal(g["idx"], h["idx"])
        f = np.random.default_rng(5).standard_normal((g["idx"].size + 1, 4))
        Pg, Ph = g["rows"].T @ (g["rows"] @ f), h["rows"].T @ (h["rows"] @ f)
        s0 = np.linalg.norm(h["rows"], axis=1).max()
        np.testing.assert_allclose(Pg, Ph, rtol=0, atol=1e-9 * s0 ** 2 * np.abs(f).max() * 4)
        if pos and g["m"] == 0:
            np.testing.assert_allclose(g["W"], h["W"], rtol=1e-12)
