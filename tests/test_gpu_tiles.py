"""Wide N tiles of the fused TF32x3 GEMM under the autotuner: T254 (192 latitudes,
128 degrees: four A slots in tensor memory, three ring stages), T318 (two tiles of
each), T382 (tiles of 144 and 96).  The tile and the slots do not enter the sums,
so the transforms stay the same bits."""
import numpy as np
import pytest

from gdpy import core, inputs
from helpers import rand_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,nlon,nlat", [(254, 768, 384), (318, 972, 480), (382, 1152, 576)])
def test_autotune_keeps_the_transforms(T, nlon, nlat):
    L = 8
    g = core.Dycore(T, nlon, nlat, L, *inputs.hybrid_coords(L), ntrac=1, dt=100.0, precision="tf32x3")
    st = inputs.smooth_random_state(T, L, ntrac=1, seed=3)
    g.set_state(st["vrt"], st["div"], st["tv"], st["lnps"], trc=st["trc"])
    a = rand_spec(T, 9, seed=T, slope=-1.0)
    grid = g.spectogrd(a)
    spec = g.grdtospec(grid)
    ch = g.autotune()
    assert ch["synth_tile"] % 16 == 0 and 16 <= ch["synth_tile"] <= 192
    assert ch["a_slots"] in (2, 3, 4)
    assert np.array_equal(g.spectogrd(a), grid)
    assert np.array_equal(g.grdtospec(grid), spec)
    g.advance(2)
    assert np.isfinite(g.get_state()["vrt"]).all()
