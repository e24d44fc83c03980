"""Held-Suarez forcing through the library where the layer pressure's forms
meet: few thick levels (the powers and the long series), many thin ones (the
short series), level counts off the kernel's groups of four and eight, both
states.  The reference is phy_run_hs.f90:42-77 in numpy's extended precision
on the library's own grid fields (in thin layers the difference of powers
loses more than the tolerance in double), analysed by the FP64 oracle.  FP64:
1e-12 of each tendency's largest value.  FP32: the state's rounding, 300 K
2^-24 against a departure from equilibrium of tens of kelvin, and the
transforms: 2e-5."""
import numpy as np
import pytest

from gdpy import core, inputs
from helpers import rel

pytestmark = pytest.mark.gpu


def forcing(g, ak, bk):
    X = np.longdouble
    f = lambda x: X(np.float32(x))
    kap = X(float(np.float32(287.05)) / float(np.float32(1004.6)))
    L, lat = g.nlev, g.grid_info()["lats"].astype(X)[:, None]
    ps = np.exp(g.get_grid("lnpsg")[0].astype(X))
    tv, vr, dv = (g.get_grid(k).astype(X) for k in ("tvg", "vrtg", "divg"))
    kf, ka, ks = (f(np.float32(1) / (np.float32(d) * np.float32(86400))) for d in (1, 40, 4))
    out = {k: np.zeros((L,) + ps.shape) for k in ("dtv", "dvrt", "ddiv")}
    for b in range(L):
        lo, up = X(ak[L - b]) + X(bk[L - b]) * ps, X(ak[L - 1 - b]) + X(bk[L - 1 - b]) * ps
        prs = ((lo ** kap * lo - up ** kap * up) / ((kap + 1) * (lo - up))) ** (1 / kap)
        bl = np.maximum(0, (prs / ps - f(0.7)) / (1 - f(0.7)))
        teq = (prs / X(1e5)) ** f(np.float32(2) / np.float32(7)) * (
            315 - 60 * np.sin(lat) ** 2 - 10 * np.log(prs / X(1e5)) * np.cos(lat) ** 2)
        out["dtv"][b] = (ka + (ks - ka) * bl * np.cos(lat) ** 4) * (np.maximum(200, teq) - tv[b])
        out["dvrt"][b], out["ddiv"][b] = -(bl * kf) * vr[b], -(bl * kf) * dv[b]
    return out


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 2e-5)])
@pytest.mark.parametrize("L", [3, 5, 8, 20, 67, 126])
def test_forcing(oracle_mod, prec, tol, L):
    T, nlon, nlat = 21, 64, 32
    ak, bk = inputs.hybrid_coords(L)
    g = core.Dycore(T, nlon, nlat, L, ak, bk, precision=prec)
    o = oracle_mod.Oracle(T, nlon, nlat, L, ak, bk)
    st = inputs.smooth_random_state(T, L, ntrac=0, seed=L)
    g.set_state(st["vrt"], st["div"], st["tv"], st["lnps"])
    g.getdyntend(1, inverse_only=True)
    want = forcing(g, ak, bk)
    a = g.getphytend()
    for k in ("dvrt", "ddiv", "dtv"):
        assert rel(a[k], o.grdtospec(want[k])) < tol, k
    assert np.abs(a["dlnps"]).max() == 0
