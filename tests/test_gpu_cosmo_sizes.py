"""sgl_cosmo_tables at the edges of its launch shapes: one and many cosmologies, one redshift and many, panels
that do not fill a warp, output points at both ends of the growth ODE's step grid."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(a - b) / np.maximum(np.abs(b), 1e-300))


@pytest.mark.parametrize("rows", [slice(0, 1), slice(4, 7), slice(0, 9)])
@pytest.mark.parametrize("cols", [slice(1, 2), slice(0, 14), slice(13, 14)])
def test_subsets_match_reference(rows, cols):
    """Each cosmology and redshift alone gives the reference's values (the bars of test_gpu_cosmo.py)."""
    from sgl_analytic_gb300._lib import Engine
    ref = dict(np.load(GOLDEN / "cosmo_ref.npz"))
    t = Engine(0).cosmo_tables(ref["params"][rows], ref["z"][cols], ref["M"][::20], ref["z_mf"][-1:])
    assert _rel(t["E"], ref["E"][rows, cols]) < 1e-14
    live = ref["z"][cols] > 0
    if live.any():
        assert _rel(t["chi"][:, live], ref["chi"][rows, cols][:, live]) < 1e-12
    assert _rel(t["D"], ref["D"][rows, cols]) < 1e-9
    assert _rel(t["sigmaM"], ref["sigmaM"][rows, ::20]) < 1e-9
    assert _rel(t["conc"], ref["conc"][rows, -1:, ::20]) < 1e-9


def test_growth_at_the_ends_of_the_step_grid():
    """z = 0 ends the last step, z = 1e6 lies before the first one (the start value holds); outputs inside one
    step keep their order."""
    from sgl_analytic_gb300._lib import Engine
    p = np.array([[0.674, 0.315, 0.0493, 0.811, 0.965, 3402.0, 0.0, -1.0, 0.0]])
    z = np.array([0.0, 1e-5, 2e-5, 1.0, 1e5, 9.999e5, 1e6])
    D = Engine(0).cosmo_tables(p, z, [1e12])["D"][0]
    assert D[0] == 1.0 and np.all(np.diff(D) < 0) and D[-1] > 0
    start = 1e-6 + (2.0 / 3.0) / (1.0 + 3402.0)             # y0 at a = 1e-6 over y0 today
    assert abs(D[-1] / D[-2] - start / (start + (1 / 9.999e5 - 1e-6))) < 1e-6


@pytest.mark.parametrize("Om", [1e-3, 1.0])
def test_extreme_matter_density_is_finite(Om):
    from sgl_analytic_gb300._lib import Engine
    p = np.array([[0.7, Om, 0.5 * Om, 0.8, 0.96, 3400.0, 0.0, -1.0, 0.0]])
    t = Engine(0).cosmo_tables(p, [0.5, 1.0], [1e8, 1e15])
    assert np.isfinite(t["sigmaM"]).all() and np.all(np.diff(t["sigmaM"][0]) < 0)
