"""FP64 zonal means of the eddy mode's analysis: an infinite value makes its row's
mean infinite (as the quotient by the row's length is), so the global mean of
its field is infinite with that sign; the other fields are untouched."""
import numpy as np
import pytest

from gdpy import core, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,nlon,nlat", [(42, 128, 64), (62, 192, 94), (126, 384, 190)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf])
def test_infinite_row(T, nlon, nlat, bad):
    g = core.Dycore(T, nlon, nlat, 8, *inputs.hybrid_coords(8), precision="f64_eddy")
    x = np.random.default_rng(T).standard_normal((9, nlat, nlon))
    s = g.grdtospec(x)
    x[1, 10, 3] = bad
    t = g.grdtospec(x)
    assert t[1, 0].real == bad
    keep = [0] + list(range(2, 9))
    assert np.array_equal(t[keep], s[keep])
