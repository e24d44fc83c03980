"""DCMIP simple physics in the FP64 state where its layer pressures change form:
few thick levels (powers and the long series), many thin ones (the short
series), level counts around the kernel's array sizes; condensation alone
(test 42) and with the boundary layer (43, 51).  The reference is the oracle's
column routine on the library's own grid fields with layer pressures in numpy's
extended precision (in double, thin layers' difference of powers loses more
than the tolerance: the exchange between two levels divides by the difference
of their pressures), its increments analysed by the oracle: 1e-9 of each
tendency's largest value."""
import numpy as np
import pytest

from helpers import rel
from test_gpu_dcmip import FVIRT, KAPPA, moist_pair

pytestmark = pytest.mark.gpu
DT = 300.0


def reference(oracle_mod, g, o, ak, bk, testcase):
    X = np.longdouble
    L, nlat, nlon = g.nlev, g.nlat, g.nlon
    field = lambda name: g.get_grid(name)[:L].reshape(L, -1)[::-1].T.copy()  # columns, top to bottom
    tv, q, u, v = (field(k) for k in ("tvg", "trcg", "ug", "vg"))
    ps = np.exp(g.get_grid("lnpsg").reshape(-1).astype(X))
    pint = np.asarray(ak, X) + np.asarray(bk, X) * ps[:, None]
    pu, pl = pint[:, :-1], pint[:, 1:]
    k = X(KAPPA)
    pmid = ((pl ** k * pl - pu ** k * pu) / ((k + 1) * (pl - pu))) ** (1 / k)
    lat = np.repeat(g.grid_info()["lats"], nlon)
    qmin = float(np.float32(1e-10))
    t = tv / (1 + FVIRT * np.maximum(qmin, q))
    t1, q1, u1, v1, precl = oracle_mod.simple_columns(DT, lat, t, q, u, v, pmid.astype(float), pint.astype(float),
                                                      ps.astype(float), int(testcase // 10 == 4), testcase != 42)
    tv1 = t1 * (1 + FVIRT * np.maximum(qmin, q1))
    grid = lambda x: np.ascontiguousarray(x.T[::-1]).reshape(L, nlat, nlon)
    vrt, div = o.getvrtdivspec(grid(u1 - u) / DT, grid(v1 - v) / DT)
    return {"dtv": o.grdtospec(grid(tv1 - tv) / DT), "dq": o.grdtospec(grid(q1 - q) / DT), "dvrt": vrt, "ddiv": div,
            "precip": precl.reshape(nlat, nlon) * 1000}


@pytest.mark.parametrize("testcase,ntrac", [(42, 3), (43, 3), (51, 1)])
@pytest.mark.parametrize("L", [3, 7, 32, 33, 65, 126])
def test_levels(oracle_mod, testcase, ntrac, L):
    from gdpy import inputs

    g, o = moist_pair(oracle_mod, testcase, ntrac, T=21, nlon=64, nlat=32, L=L, dt=DT)
    g.getdyntend(3, inverse_only=True)
    a = g.getphytend()
    b = reference(oracle_mod, g, o, *inputs.hybrid_coords(L), testcase)
    for k in ("dvrt", "ddiv", "dtv"):
        assert rel(a[k], b[k]) < 1e-9, k
    assert rel(a["dtrc"][0], b["dq"]) < 1e-9
    assert rel(g.get_grid("precip"), b["precip"]) < 1e-9
