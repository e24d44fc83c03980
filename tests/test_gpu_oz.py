"""The plain FP64 Legendre GEMMs on the tensor cores (operands split into exact
8-bit digits) at the edges of their tiles: latitude and degree counts around
the 16-column step and the 32-column tile, contractions around the 32-deep
chunk and the 128-deep segment, columns around the 128-column tile, orders
with a single degree; columns of very different size side by side; infinities
and NaN.  Against the FP64 oracle at the plain path's 1e-12 of each field's
largest value."""
import numpy as np
import pytest

from gdpy import core, inputs
from helpers import rand_spec, rel

pytestmark = pytest.mark.gpu


def pair(oracle_mod, T, nlon, nlat, L=64):
    g = core.Dycore(T, nlon, nlat, L, *inputs.hybrid_coords(L))
    return g, oracle_mod.Oracle(T, nlon, nlat, 4, *inputs.hybrid_coords(4))


@pytest.mark.parametrize("T,nlon,nlat,nb", [(1, 8, 4, 1), (15, 48, 30, 31), (31, 96, 62, 32), (32, 108, 64, 33),
                                            (63, 192, 94, 64), (64, 216, 130, 65), (66, 216, 100, 40),
                                            (128, 432, 256, 2), (131, 432, 258, 3), (170, 512, 256, 5)])
def test_transforms(oracle_mod, T, nlon, nlat, nb):
    g, o = pair(oracle_mod, T, nlon, nlat)
    a, b = rand_spec(T, nb, seed=T, slope=-1.0), rand_spec(T, nb, seed=T + 1, slope=-1.0)
    grid = o.spectogrd(a)
    assert rel(g.spectogrd(a), grid) < 1e-12
    assert rel(g.grdtospec(grid), o.grdtospec(grid)) < 1e-12
    for x, y in zip(g.getuv(a, b), o.getuv(a, b)):
        assert rel(x, y) < 1e-12
    u, v = o.getuv(a, b)
    for x, y in zip(g.getvrtdivspec(u, v), o.getvrtdivspec(u, v)):
        assert rel(x, y) < 1e-12
    for x, y in zip(g.getgrad(a), o.getgrad(a)):
        assert rel(x, y) < 1e-12


def test_columns_keep_their_own_scale(oracle_mod):
    # every column has an exponent of its own: fields 1e-200 to 1e200 in one call,
    # each to 1e-12 of itself, and a zero field stays zero
    T, nlon, nlat = 42, 128, 64
    g, o = pair(oracle_mod, T, nlon, nlat, 20)
    a = rand_spec(T, 8, seed=5, slope=-1.0)
    scale = 10.0 ** np.array([-200, -100, -30, -3, 0, 40, 120, 200])
    x = g.spectogrd(np.concatenate([a * scale[:, None], np.zeros((1, g.nlm))]))
    y = o.spectogrd(a)
    for k in range(8):
        assert rel(x[k] / scale[k], y[k]) < 1e-12
    assert np.all(x[8] == 0)
    s = g.grdtospec(y * scale[:, None, None])
    t = o.grdtospec(y)
    for k in range(8):
        assert rel(s[k] / scale[k], t[k]) < 1e-12


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_bad_values_stay_visible(bad):
    # an infinity or NaN makes its own field non-finite and leaves the others alone
    T, nlon, nlat = 42, 128, 64
    g = core.Dycore(T, nlon, nlat, 20, *inputs.hybrid_coords(20))
    a = rand_spec(T, 3, seed=9)
    y = g.spectogrd(a)
    a[1, 60] = bad
    x = g.spectogrd(a)
    assert not np.isfinite(x[1]).any()
    assert np.array_equal(x[[0, 2]], y[[0, 2]])
    y[1, 10, 3] = bad
    s = g.grdtospec(y)
    assert not np.isfinite(s[1]).any() and np.isfinite(s[[0, 2]]).all()


@pytest.mark.parametrize("T,nlon,nlat,nb", [(1, 8, 4, 1), (42, 128, 64, 21)])
def test_fp64_pipe(oracle_mod, monkeypatch, T, nlon, nlat, nb):
    # contexts whose digits take too much memory keep the FP64 pipe
    monkeypatch.setenv("GD_FP64_TC_GB", "0")
    g, o = pair(oracle_mod, T, nlon, nlat, 20)
    a = rand_spec(T, nb, seed=T, slope=-1.0)
    grid = o.spectogrd(a)
    assert rel(g.spectogrd(a), grid) < 1e-12
    assert rel(g.grdtospec(grid), o.grdtospec(grid)) < 1e-12
    for x, y in zip(g.getuv(a, a), o.getuv(a, a)):
        assert rel(x, y) < 1e-12
