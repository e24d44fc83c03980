"""Dynamics tendencies of the FP64 state around the level counts where the
column kernel changes its levels per warp (32 / 33, 64 / 65), with blocks that
are full, short by one and of one level, against the FP64 oracle.  The oracle's
alfa = 1 - p0 / dp ln(p1 / p0) loses up to 1 / (dp / p) of a thin layer's digits,
a factor of 100 at 65 levels, and the pressure gradient sums them: 1e-11 of each
tendency's largest value."""
import pytest

from gdpy import core, inputs
from helpers import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [31, 32, 33, 40, 47, 64, 65])
def test_tendencies(oracle_mod, L):
    T, nlon, nlat, nt = 21, 108, 54, 2
    ak, bk = inputs.hybrid_coords(L)
    g = core.Dycore(T, nlon, nlat, L, ak, bk, ntrac=nt)
    o = oracle_mod.Oracle(T, nlon, nlat, L, ak, bk, ntrac=nt)
    st = inputs.smooth_random_state(T, L, ntrac=nt, seed=L)
    for m in (g, o):
        m.set_state(st["vrt"], st["div"], st["tv"], st["lnps"], trc=st["trc"])
    a, b = g.getdyntend(1), o.getdyntend(1)
    for k in ("dvrt", "ddiv", "dtv", "dtrc", "dlnps"):
        assert rel(a[k], b[k]) < 1e-11, k
