"""Order 0 of the split modes (the zonal means, on the IEEE path): zonally
symmetric fields through every transform of the FP64-state split modes
against the FP64 oracle, at row counts and contraction lengths off the
kernels' tiles (8 rows, 32 columns, chunks of 64 and 32).  Orders m >= 1 are
zero here, so the FP64 tolerance of the plain path holds: 1e-12 of the
largest value."""
import numpy as np
import pytest

from gdpy import core, inputs
from helpers import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64_tf32x3", "f64_eddy"])
@pytest.mark.parametrize("T,nlon,nlat,nb", [(21, 64, 32, 1), (62, 192, 94, 33), (63, 192, 98, 32), (64, 216, 100, 40),
                                            (127, 384, 194, 3)])
def test_zonal_fields(oracle_mod, prec, T, nlon, nlat, nb):
    ak, bk = inputs.hybrid_coords(64)
    g = core.Dycore(T, nlon, nlat, 64, ak, bk, precision=prec)
    o = oracle_mod.Oracle(T, nlon, nlat, 4, *inputs.hybrid_coords(4))
    rng = np.random.default_rng(T + nb)
    a, b = np.zeros((2, nb, g.nlm), np.complex128)
    a[:, : T + 1] = rng.standard_normal((nb, T + 1)) / np.arange(1, T + 2)
    b[:, : T + 1] = rng.standard_normal((nb, T + 1)) / np.arange(1, T + 2)
    a[:, 0] += 280.0
    grid = o.spectogrd(a)
    assert rel(g.spectogrd(a), grid) < 1e-12
    assert rel(g.grdtospec(grid), a) < 1e-12
    uo, vo = o.getuv(a, b)
    u, v = g.getuv(a, b)
    assert rel(u, uo) < 1e-12 and rel(v, vo) < 1e-12
    vrt, div = g.getvrtdivspec(uo, vo)
    vrto, divo = o.getvrtdivspec(uo, vo)
    assert rel(vrt, vrto) < 1e-12 and rel(div, divo) < 1e-12
    gx, gy = g.getgrad(a)
    ox, oy = o.getgrad(a)
    assert np.abs(gx).max() == np.abs(ox).max() == 0.0 and rel(gy, oy) < 1e-12
