"""The semi-implicit stage's running sums over the levels: one step through
the library against the FP64 oracle at level counts around the sixteen level
blocks of a coefficient (fewer levels than blocks, one level per block, a
short last block, the most levels).  1e-10 of each field's largest value: with
126 levels the oracle's own alfa = 1 - pk/dpk ln(pk1/pk) loses p/dp ~ 6400
units of rounding (7e-13) in the pressure gradient, and the divergence is one
to two orders below the terms that make it.  The FP32 state takes the FP64
state's step to 1e-4 (vorticity, divergence), its rounding in the balanced terms."""
import numpy as np
import pytest

from gdpy import core, inputs
from helpers import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("explicit", [False, True])
@pytest.mark.parametrize("L", [3, 15, 16, 17, 33, 64, 126])
def test_one_step(oracle_mod, L, explicit):
    T, nlon, nlat, dt = 21, 64, 32, 300.0 if explicit else 1200.0
    ak, bk = inputs.hybrid_coords(L)
    st = inputs.smooth_random_state(T, L, ntrac=1, seed=L)
    out = {}
    o = oracle_mod.Oracle(T, nlon, nlat, L, ak, bk, ntrac=1, dt=dt, explicit=explicit)
    g = core.Dycore(T, nlon, nlat, L, ak, bk, ntrac=1, dt=dt, explicit=explicit)
    f = core.Dycore(T, nlon, nlat, L, ak, bk, ntrac=1, dt=dt, explicit=explicit, precision="fp32")
    for name, m in (("o", o), ("g", g), ("f", f)):
        m.set_state(st["vrt"], st["div"], st["tv"], st["lnps"], trc=st["trc"])
        m.advance(1)
        out[name] = m.get_state()
    for k in ("vrt", "div", "tv", "trc", "lnps"):
        assert rel(out["g"][k], out["o"][k]) < 1e-10, k
    for k, tol in (("vrt", 1e-4), ("div", 1e-4), ("tv", 1e-5), ("trc", 1e-5), ("lnps", 1e-5)):
        assert rel(out["f"][k], out["g"][k]) < tol, k
