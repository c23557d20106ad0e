"""The mixed path's vp kernels at the edges of their tiles (16 k x 112 q, 32 cells, pieces of a shell; chains of 32
points), against the FP64 path: the bar of test_gpu_vp.py, 2e-8 (1 + |ln R|)."""
import numpy as np
import pytest

from tests.conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _closure(shells):
    """The first `shells` shells of the golden sub-closure."""
    d = dict(np.load(GOLDEN / "vp_zs1_sub.npz"))
    g = int(d["sh_g"][shells])
    c = int(d["gstart"][g])
    return dict(d, K=d["K"][:shells - 1], sh_g=d["sh_g"][:shells + 1], gstart=d["gstart"][:g + 1], cu=d["cu"][:c],
                cw=d["cw"][:c], **{k: d[k][:g] for k in ("ga", "gb", "gc", "glo", "ghi")})


def _compare(d, k, q):
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
    e = Engine(0)
    e.set_vp(d)
    a, b = e.vp_lnR(k, q, SGL_FP64), e.vp_lnR(k, q, SGL_MIXED)
    dre, dim = np.abs(a.real - b.real), np.abs(a.imag - b.imag)
    dim = np.minimum(dim, np.abs(dim - 2 * np.pi))                     # principal branch
    assert np.all(np.maximum(dre, dim) <= 2e-8 * (1 + np.abs(a)))


@pytest.mark.parametrize("nk,nq", [(7, 112), (8, 31), (8, 32), (15, 111), (16, 112), (17, 113), (33, 225), (61, 40)])
@pytest.mark.parametrize("shells", [1, 2, 6])
def test_grid_sizes(nk, nq, shells):
    _compare(_closure(shells), np.linspace(0.0, 1010.0, nk), np.linspace(0.0, 800.0, nq))


def test_right_clipped_and_linear_runs():
    """Every rate interval mirrored (right runs), every third group linear, runs of a few cells."""
    d = _closure(3)
    ns = d["u"].size
    clipped = d["gc"] != 0
    m = dict(d, K=d["K"][:, ::-1, ::-1].copy(), w=d["w"][::-1].copy(), ga=-d["ga"],
             glo=np.where(clipped, ns - 1 - d["ghi"], d["glo"]).astype(np.int32),
             ghi=np.where(clipped, ns - 1 - d["glo"], d["ghi"]).astype(np.int32))
    _compare(m, np.linspace(0.0, 900.0, 20), np.linspace(0.0, 700.0, 50))


def test_large_phases_take_the_fp64_sine():
    """Weights scaled up until Im z passes the float-float sine's 2e4."""
    d = _closure(2)
    big = dict(d, cw=d["cw"] * 2e3)
    from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
    e = Engine(0)
    e.set_vp(big)
    k, q = np.linspace(0.0, 3.0, 16), np.linspace(0.0, 2.0, 40)
    a, b = e.vp_lnR(k, q, SGL_FP64), e.vp_lnR(k, q, SGL_MIXED)
    assert np.all(np.abs(np.exp(a - b) - 1) <= 1e-5 + 2e-8 * np.abs(a))


@pytest.mark.parametrize("n", [1, 2, 20, 31, 32, 33, 608, 609])
@pytest.mark.parametrize("shells", [1, 6])
@pytest.mark.parametrize("axis", ["k", "q"])
def test_lines_of_points(n, shells, axis):
    """The probes' lines: part of a warp, whole warps, the last count that takes the line kernel and the next."""
    x = np.geomspace(1.0, 900.0, n)
    d = _closure(shells)
    if axis == "k":
        _compare(d, x, np.zeros(1))
        _compare(d, x, np.full(1, 300.0))
    else:
        _compare(d, np.zeros(1), x)


def test_lines_of_right_and_linear_runs():
    d = _closure(3)
    ns = d["u"].size
    clipped = d["gc"] != 0
    m = dict(d, K=d["K"][:, ::-1, ::-1].copy(), w=d["w"][::-1].copy(), ga=-d["ga"],
             glo=np.where(clipped, ns - 1 - d["ghi"], d["glo"]).astype(np.int32),
             ghi=np.where(clipped, ns - 1 - d["glo"], d["ghi"]).astype(np.int32))
    _compare(m, np.linspace(0.0, 900.0, 20), np.full(1, 40.0))
    _compare(m, np.full(1, 90.0), np.linspace(0.0, 700.0, 50))
