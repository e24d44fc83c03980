"""The closure net's tensor-core chain at the edges of its tiles: widths
around the 16-column MMA step, the 64-input weight chunk and the 128-output
half, first layers wider than one 256-input pass, batches around the 128-row
tile and the transposing kernel's 128-column block, one hidden layer and
several.  Against the float64 oracle with the same BF16-rounded weights:
outputs 1e-5, gradients 1e-4 of each block's largest entry (FP32 accumulation
over at most a few hundred terms, and over the batch)."""
import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 1, 1, 1), (5, 16, 1, 3), (31, 40, 2, 17), (64, 64, 3, 64), (193, 128, 2, 192), (100, 130, 2, 129),
          (256, 256, 4, 256), (193, 200, 1, 65)]


def make(shape, n, seed):
    import mlp_oracle as mo
    from gdpy import core

    rng = np.random.default_rng(seed)
    net = core.Mlp(*shape, seed=1)
    shp = mo.shapes(*shape)
    p = np.concatenate([np.concatenate([rng.standard_normal(fo * fi) * np.sqrt(2.0 / fi),
                                        rng.standard_normal(fo) * 0.1]) for fo, fi in shp]).astype(np.float32)
    net.set_params(p)
    x = rng.standard_normal((n, shape[0])).astype(np.float32)
    t = rng.standard_normal((n, shape[3])).astype(np.float32)
    return mo, net, shp, p, x, t


@pytest.mark.parametrize("n", [1, 127, 129, 1000])
@pytest.mark.parametrize("shape", SHAPES + [(257, 64, 2, 30), (379, 256, 2, 200), (520, 96, 1, 8)])
def test_forward(shape, n):
    mo, net, shp, p, x, _ = make(shape, n, n)
    y = net.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    assert rel(y, mo.forward(p, shp, x)[0]) < 1e-5


@pytest.mark.parametrize("n", [1, 33, 128, 700])
@pytest.mark.parametrize("shape", SHAPES)
def test_gradient(shape, n):
    mo, net, shp, p, x, t = make(shape, n, n)
    loss, g = net.loss_grad(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    lo, go = mo.loss_grad(p, shp, x, t)
    assert abs(loss - lo) <= 1e-5 * lo
    o = 0
    for fo, fi in shp:
        for sz in (fo * fi, fo):
            assert rel(g[o:o + sz], go[o:o + sz]) < 1e-4, (fo, fi, sz)
            o += sz


def test_updated_weights_are_read():
    # a training step repacks the weights: the next forward pass uses them
    mo, net, shp, p, x, t = make((31, 40, 2, 17), 300, 3)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    for _ in range(2):
        net.train_step(xd, td, 1e-2)
    q = net.get_params()
    assert not np.array_equal(p, q)
    assert rel(net.forward(xd).cpu().numpy(), mo.forward(q, shp, x)[0]) < 1e-5
