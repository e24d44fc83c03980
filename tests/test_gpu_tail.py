"""FP32 transforms whose last two columns go beside the tensor-core GEMM: column
counts with and without such a rest (nb = 64, 65, 66 fields), latitude counts
off the warp's four rows, degree counts off the 32 lanes and the 128-degree
blocks.  Against the FP64 oracle: the last of 65 fields at 2e-5 of its largest
value, the FP32 path's tolerance, the others at their mode's."""
import pytest

from gdpy import core, inputs
from helpers import rand_spec, rel

pytestmark = pytest.mark.gpu


SPLIT_TOL = {"tf32x3": 2e-5, "bf16x3": 2e-4}  # of the GEMM columns, as for the modes elsewhere


@pytest.mark.parametrize("T,nlon,nlat,nb", [(150, 486, 228, 65), (161, 486, 250, 65), (170, 512, 256, 64),
                                            (170, 512, 256, 65), (170, 512, 256, 66)])
@pytest.mark.parametrize("precision", ["tf32x3", "bf16x3"])
def test_transforms(oracle_mod, T, nlon, nlat, nb, precision):
    g = core.Dycore(T, nlon, nlat, 64, *inputs.hybrid_coords(64), precision=precision)
    o = oracle_mod.Oracle(T, nlon, nlat, 4, *inputs.hybrid_coords(4))

    def close(x, y):
        assert rel(x, y) < SPLIT_TOL[precision]
        assert rel(x[-1], y[-1]) < (2e-5 if nb == 65 else SPLIT_TOL[precision])

    a, b = rand_spec(T, nb, seed=T, slope=-1.0), rand_spec(T, nb, seed=T + 1, slope=-1.0)
    grid = o.spectogrd(a)
    close(g.spectogrd(a), grid)
    close(g.grdtospec(grid), a)
    u, v = o.getuv(a, b)
    for x, y in zip(g.getuv(a, b), (u, v)):
        close(x, y)
    for x, y in zip(g.getgrad(a), o.getgrad(a)):
        close(x, y)
    for x, y in zip(g.getvrtdivspec(u, v), (a, b)):
        assert rel(x[:, 1:], y[:, 1:]) < SPLIT_TOL[precision]  # 130 fields' columns: no rest
