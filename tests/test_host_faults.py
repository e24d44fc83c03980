"""What the host code does when a call of the CUDA runtime fails and the order
in which it hands work to the device, on a runtime without a GPU
(fake_runtime.py)."""
import pytest

import fake_runtime


@pytest.mark.parametrize("hidden", [16, 300])  # the tensor-core and the SIMT training path
def test_training_after_a_failed_allocation(hidden):
    """A training batch whose buffers do not fit is refused and leaves the net as
    it was: the next smaller batch runs on the buffers it had (or gets its own),
    the same batch runs once there is memory."""
    fake_runtime.run(r"""
H, SMALL, BIG, NOUT = %d, 128, 40000, 3
rt.fake_watch(b"k_mse", 3)  # the output gradient's buffer
x, t = device(4 * BIG * 5), device(4 * BIG * NOUT)

def net():
    h = vp()
    assert lib.gd_mlp_init(5, H, 2, NOUT, 1, 0, ctypes.byref(h)) == 0
    return h

def grad(h, n):
    # status, device memory it took, where the output gradient went, kernels
    before = rt.fake_used()
    log()
    rc = lib.gd_mlp_loss_grad(h, x, t, n, None, None)
    l = log()
    gy = [p for w, p, _, _ in l if w.startswith("launch:") and "5k_mse" in w and "final" not in w]
    return rc, rt.fake_used() - before, gy, sum(w.startswith("launch:") for w, _, _, _ in l)

h = net()
_, small, _, n_small = grad(h, SMALL)
lib.gd_mlp_destroy(h)
for trained in (False, True):
    k = 0
    while True:
        h = net()
        gy0 = grad(h, SMALL)[2] if trained else None
        rt.fake_fail(k)
        rc, kept, gy, n = grad(h, BIG)
        rt.fake_fail(-1)
        if rc == 0:
            break
        assert rc == core.GD_ERR_CUDA and n == 0 and kept == 0, (k, rc, n, kept)
        rc, took, gy, n = grad(h, SMALL)
        assert rc == 0 and n == n_small, (k, rc, n)
        assert gy == gy0 if trained else took == small, (k, took)
        rc, took, gy, n = grad(h, BIG)
        assert rc == 0 and took > 0 and gy != gy0, (k, rc, took)
        lib.gd_mlp_destroy(h)
        k += 1
    assert k >= (6 if H > 256 else 14), k  # every buffer's allocation was made to fail
""" % hidden)


@pytest.mark.parametrize("fused", ["1", "0"])
def test_uploads_are_ordered_with_the_kernels_that_read_them(fused):
    """Tables and parameters are copied in the order of the stream that reads
    them: whatever goes through the legacy default stream has completed before
    a kernel starts on another stream, which would not wait for it."""
    fake_runtime.run(r"""
T, nlon, nlat, L = 21, 64, 32, 8
ak, bk = inputs.hybrid_coords(L)
st = inputs.hs_rest_state(T, L, seed=0)
for mode in core.PREC:
    p = vp()
    assert lib.gd_pattern_init(500e3, 1200.0, 21600.0, 0.5, 1, nlon, nlat, T, 1.0, 1, 0, ctypes.byref(p)) == 0
    assert lib.gd_pattern_start(p) == 0
    g = core.Dycore(T, nlon, nlat, L, ak, bk, dt=1200.0, precision=mode)
    g.set_state(st["vrt"], st["div"], st["tv"], st["lnps"])
    assert lib.gd_set_sppt(g.h, p, 0.05, 0.1) == 0
    g.advance(3)
    s = np.zeros((3, g.nlm), complex)
    g.getvrtdivspec(*g.getuv(s, s))
    g.getgrad(g.grdtospec(g.spectogrd(s)))
    g.close()
for shape in ((5, 16, 2, 3), (5, 300, 2, 3)):
    h, n = vp(), ctypes.c_longlong()
    assert lib.gd_mlp_init(*shape, 1, 0, ctypes.byref(h)) == 0
    lib.gd_mlp_nparams(h, ctypes.byref(n))
    q = [ptr(np.ones(k, np.float32)) for k in (n.value, 5, 5, 3, 3)]
    assert lib.gd_mlp_set_params(h, q[0]) == 0 and lib.gd_mlp_set_norm(h, *q[1:]) == 0
    x, t = device(4 * 5 * 1000), device(4 * 3 * 1000)
    assert lib.gd_mlp_train_step(h, x, t, 1000, 1e-3, None) == 0
l = log()
assert sum(w == "h2d" for w, _, _, _ in l) > 50
pending = None
for w, p, n, s in l:
    if w in ("h2d", "memset") and s == 0:
        pending = (w, n)
    elif w == "sync" and s == 0:
        pending = None
    elif w.startswith("launch:") and s != 0:
        assert pending is None, (pending, w)
""", {"GD_TC_FUSED": fused})


@pytest.mark.parametrize("mode", ["fp64", "tf32x3", "f64_eddy"])
def test_a_wait_that_gave_up_is_raised_by_the_call_that_ran_it(mode):
    """A bounded wait of the tensor-core Legendre kernels that gives up leaves a
    code in the context's error flag: every entry point that hands out results
    raises it, once."""
    fake_runtime.run(r"""
T, nlon, nlat, L = 42, 128, 64, 8
ak, bk = inputs.hybrid_coords(L)
st = inputs.hs_rest_state(T, L, seed=0)
log()
g = core.Dycore(T, nlon, nlat, L, ak, bk, dt=1200.0, precision="%s")
flag, = [p for w, p, n, _ in log() if w == "register"]
g.set_state(st["vrt"], st["div"], st["tv"], st["lnps"])
s, s1 = np.zeros((3, g.nlm), complex), np.zeros((3, g.nlm), np.complex64)
x, x1 = np.zeros((3, nlat, nlon)), np.zeros((3, nlat, nlon), np.float32)
feat = np.zeros((nlat * nlon, 3 * L + 1), np.float32)
calls = dict(spectogrd=lambda: g.spectogrd(s), spectogrd_f=lambda: g.spectogrd(s1), grdtospec=lambda: g.grdtospec(x),
             grdtospec_f=lambda: g.grdtospec(x1), getuv=lambda: g.getuv(s, s), getuv_f=lambda: g.getuv(s1, s1),
             getvrtdivspec=lambda: g.getvrtdivspec(x, x), getvrtdivspec_f=lambda: g.getvrtdivspec(x1, x1),
             getgrad=lambda: g.getgrad(s), getgrad_f=lambda: g.getgrad(s1), getdyntend=lambda: g.getdyntend(1),
             getphytend=lambda: g.getphytend(), inverse=lambda: g.getdyntend(1, inverse_only=True),
             get_state=lambda: g.get_state(), get_grid=lambda: g.get_grid("ug"), diag=lambda: g.diag(),
             features=lambda: g._chk(lib.gd_closure_features(g.h, ptr(feat))), sync=lambda: g.sync())
for name, f in calls.items():
    f()
    ctypes.memset(flag, 54, 1)
    try:
        f()
    except core.GdError as e:
        assert e.code == core.GD_ERR_CUDA and "gave up" in str(e), (name, e)
    else:
        raise AssertionError(name + " returned")
    f()
""" % mode)


def test_digits_leave_room_for_other_contexts():
    """The digits of the plain FP64 mode are there for speed: contexts take them
    while half of the device stays free, and what fits without them in half of
    the device fits with them."""
    fake_runtime.run(r"""
ak, bk = inputs.hybrid_coords(20)

def fill(total):
    # contexts until one does not fit: device memory each took, with digits or not
    rt.fake_total(total)
    out, keep = [], []
    while True:
        log()
        before = rt.fake_used()
        try:
            keep.append(core.Dycore(42, 128, 64, 20, ak, bk, dt=1200.0))
        except core.GdError as e:
            assert e.code == core.GD_ERR_NOMEM
            for g in keep:
                g.close()
            return out
        out.append((rt.fake_used() - before, any("k_oz_table" in w for w, _, _, _ in log())))
        assert not out[-1][1] or total - rt.fake_used() >= total // 2

big = 1 << 30
with_digits = fill(big)
assert with_digits[0][1] and not with_digits[-1][1]
plain = with_digits[-1][0]
assert len(with_digits) >= big // 2 // plain, (len(with_digits), plain)
""")


def test_a_context_gives_its_digits_back_for_what_it_must_have():
    """An allocation of a context that only fits without the context's digits
    gets their memory; the context goes on on the FP64 pipe."""
    fake_runtime.run(r"""
ak, bk = inputs.hybrid_coords(20)
st = inputs.hs_rest_state(42, 20, seed=0)
rt.fake_total(1 << 30)

def kernels(f):
    log()
    f()
    l = [w for w, _, _, _ in log() if w.startswith("launch:")]
    return any("k_oz_gemm" in w for w in l), any("k_synthI" in w or "k_analI" in w for w in l)

for step in (0, 1, 3):
    g = core.Dycore(42, 128, 64, 20, ak, bk, dt=1200.0)
    g.set_state(st["vrt"], st["div"], st["tv"], st["lnps"])
    g.advance(step)
    assert kernels(g.getphytend) == (True, False)
    used, rest = rt.fake_used(), device((1 << 30) - rt.fake_used() - 4096)
    s = np.zeros((70, g.nlm), complex)
    assert kernels(lambda: g.getuv(s, s)) == (False, True)
    rt.cudaFree(rest)
    assert rt.fake_used() < used
    assert kernels(lambda: g.advance(1)) == (False, True)
    assert kernels(g.getphytend) == (False, True)
    assert kernels(lambda: g.grdtospec(np.zeros((3, 64, 128)))) == (False, True)
    g.advance(3)
    g.close()
""")


def test_a_failed_call_does_not_fail_the_next_one():
    """An allocation that fails is reported by its own call: the same call
    afterwards, with memory there, runs."""
    fake_runtime.run(r"""
ak, bk = inputs.hybrid_coords(8)
for mode in ("fp64", "fp32", "tf32x3"):
    for k in range(8):
        g = core.Dycore(21, 64, 32, 8, ak, bk, dt=1200.0, precision=mode)
        s = np.zeros((3, g.nlm), complex)
        rt.fake_fail(k)
        try:
            g.getuv(s, s)
        except core.GdError as e:
            assert e.code == core.GD_ERR_CUDA
        rt.fake_fail(-1)
        g.getuv(s, s)
        g.close()
""")


def test_a_context_that_cannot_be_made_leaves_nothing():
    """Whichever allocation of gd_init fails, all memory taken before it is given back."""
    fake_runtime.run(r"""
ak, bk = inputs.hybrid_coords(8)
for mode in core.PREC:
    for T, nlon, nlat in ((21, 64, 32), (42, 128, 64)):
        k = 0
        while True:
            rt.fake_fail(k)
            try:
                g = core.Dycore(T, nlon, nlat, 8, ak, bk, dt=1200.0, precision=mode)
            except core.GdError:
                assert rt.fake_used() == 0, (mode, k, rt.fake_used())
            else:
                failed = any(w == "nomem" for w, _, _, _ in log())  # the digits are the one optional allocation
                g.close()
                assert rt.fake_used() == 0
                if not failed:
                    break
            rt.fake_fail(-1)
            k += 1
        rt.fake_fail(-1)
        assert k > 50
""")


def test_a_call_that_fails_leaves_no_copy_in_flight():
    """A transform in several chunks that fails in one of them has waited for the
    copies of the chunks before it when it returns."""
    fake_runtime.run(r"""
ak, bk = inputs.hybrid_coords(8)
for mode in ("fp64", "fp32", "tf32x3"):
    for k in range(12):
        g = core.Dycore(21, 64, 32, 8, ak, bk, dt=1200.0, precision=mode)
        s, x = np.zeros((50, g.nlm), complex), np.zeros((50, 32, 64))
        for f in (lambda: g.getuv(s, s), lambda: g.getvrtdivspec(x, x)):
            log()
            rt.fake_fail(k)
            try:
                f()
            except core.GdError:
                pass
            rt.fake_fail(-1)
            l = log()
            copies = [i for i, (w, _, n, _) in enumerate(l) if w in ("h2d", "d2h")]
            stream = l[copies[-1]][3] if copies else 0
            assert not copies or ("sync", 0, 0, stream) in l[copies[-1]:], (mode, k, l[copies[-1]:])
        g.close()
""")


def test_results_are_copied_to_pages_that_are_there():
    """The transforms' results go to the caller's arrays in pages that the host has
    brought into being: the device faults new pages one by one."""
    fake_runtime.run(r"""
ak, bk = inputs.hybrid_coords(20)
for mode in ("fp64", "tf32x3"):
    g = core.Dycore(42, 128, 64, 20, ak, bk, dt=1200.0, precision=mode)
    keep = []
    for nb in (3, 20, 65):
        s = np.zeros((nb, g.nlm), complex)
        log()
        keep += [g.getgrad(s), g.getuv(s, s), g.spectogrd(s)]
        l = log()
        assert any(w == "d2h" for w, _, _, _ in l) and not any(w == "absent" for w, _, _, _ in l), nb
""")
