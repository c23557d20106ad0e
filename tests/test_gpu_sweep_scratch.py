"""The FP64 separable sweep on more cells than its half-angle table may hold (2^21: 1 GiB): no table, the same ln Phi."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


def test_many_cells_take_no_table():
    """Every cell 30 times with a thirtieth of its weight: 2.39 M cells.  63 rows never take the table, 65 would: the second
    call may grow the engine's buffers (1.6 GB) by 65 / 63 and their rounding, not by the 1.22 GB of half angles."""
    import torch
    from sgl_analytic_gb300 import Lam, Population
    pop = Population.load(GOLDEN / "pop_zs1_sub.npz")
    kk, kg = np.linspace(0.0, 900.0, 65), np.linspace(0.0, 700.0, 3200)
    one = Lam(pop, xi=False)(kk, kg)
    m = 30
    pop.k0, pop.g0, pop.ig, pop.w0 = (np.repeat(a, m) for a in (pop.k0, pop.g0, pop.ig, pop.w0 / m))
    lam = Lam(pop, xi=False)
    lam(kk[:63], kg)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    many = lam(kk, kg)
    free1 = torch.cuda.mem_get_info()[0]
    assert np.all(np.abs(many - one) <= np.maximum(1e-10, 1e-12 * np.abs(one)))
    assert free0 - free1 < 2 ** 29
