"""An instance's ln Phi has the same bits in whatever batch it is solved: alone (its cells cut into many parts), beside
instances that take some of the chip, and beside one whose k tiles fill it (nothing is cut)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [2048, 2049, 4096 + 511, 70000, 64 * 2048 + 1, 200001])
@pytest.mark.parametrize("precision", [0, 1])
def test_bits_do_not_depend_on_the_batch(cells, precision):
    from sgl_analytic_gb300._lib import Engine
    rng = np.random.default_rng(cells)
    kap, w = np.exp(rng.uniform(-5, 0, cells)), np.exp(rng.uniform(-4, 1, cells))
    nk = 129
    got = []
    for beside in (0, 130_000, 400_000, 1_500_000):                       # k points of a second instance of 5 cells
        two = beside > 0
        e = Engine(0)
        e.cfb_set(dict(inst_plane0=[0, 1, 2][:2 + two], plane_cells=[0, cells, cells + 5][:2 + two],
                       kap=np.concatenate([kap, np.full(5 * two, 0.1)]), w=np.concatenate([w, np.ones(5 * two)]),
                       nk=[nk, beside][:1 + two], dk=[0.37, 1e-3][:1 + two], closure=[0] * (1 + two),
                       V=[0.3, 0.0][:1 + two], nstate=0, vp_D=np.zeros(1 + two), vp_K=np.zeros(1), vp_w=np.zeros(1)))
        got.append(e.cfb_lnphi(precision)[:nk])
    for g in got[1:]:
        assert np.array_equal(g, got[0])
