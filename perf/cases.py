"""Performance cases of the dycore: what a host model, a driver or a notebook has the library do.

Three kinds of calls, each through a public entry point:

* ``forecast`` -- the host-model call sequence gd_set_state, gd_advance, gd_get_state over page-locked host arrays
  (double, or single precision as the reference's default build has them): a few time steps from a new initial
  state, at the configurations of the benchmark and the tests;
* ``transform`` -- the spherical-harmonic facade (spectogrd, grdtospec, getuv, getvrtdivspec, getgrad) on ordinary
  host arrays;
* ``closure`` -- the per-column network: inference over a grid's columns, and the loss and gradient of a minibatch.

Initial states are seeded: eddies of every wavenumber on a stratified atmosphere, correlated in the vertical
(vorticity amplitudes falling as n^(-2/3), divergence as n^(-1/3), temperature, ln ps and tracers as 1/n^2).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gfs-dycore_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from gdpy import core  # noqa: E402


def _forecast(name, T, nlon, nlat, L, nt, prec, dt, steps, physics="hs"):
    return dict(name=name, kind="forecast", T=T, nlon=nlon, nlat=nlat, L=L, nt=nt, prec=prec, dt=dt, steps=steps,
                physics=physics)


def _transform(name, op, T, nlon, nlat, nb, prec, single):
    return dict(name=name, kind="transform", op=op, T=T, nlon=nlon, nlat=nlat, nb=nb, prec=prec, single=single)


def _closure(name, op, L, hidden, layers, cols):
    return dict(name=name, kind="closure", op=op, L=L, hidden=hidden, layers=layers, cols=cols)


def listed():
    return [
        # the Held-Suarez test-bed: half a day of the smallest model, plain FP64 (the default precision)
        _forecast("hs_t42l20_fp64", 42, 128, 64, 20, 0, "fp64", 1200.0, 36),
        # the medium plain FP64 configuration with three tracers: one hour
        _forecast("hs_t126l64_fp64", 126, 384, 190, 64, 3, "fp64", 600.0, 6),
        # a host model that exchanges the state every step (the benchmark's end-to-end line), at the truncation of
        # a coarse ensemble member, tensor-core path
        _forecast("hs_t62l64_tf32x3", 62, 192, 94, 64, 3, "tf32x3", 1200.0, 1),
        # the same at the truncation of a fine member
        _forecast("hs_t254l64_tf32x3", 254, 768, 384, 64, 3, "tf32x3", 300.0, 1),
        # the same at the headline operational size, four tracers
        _forecast("hs_t574l64_tf32x3", 574, 1152, 576, 64, 4, "tf32x3", 150.0, 1),
        # an accurate run on an FP64 state with the eddies on the tensor cores; single-precision history output
        _forecast("hs_t254l64_f64_eddy", 254, 768, 384, 64, 3, "f64_eddy", 300.0, 3),
        # moist run with the simple physics (condensation, surface fluxes, boundary-layer diffusion): half an hour
        _forecast("moist_t126l64_f64_eddy", 126, 384, 190, 64, 3, "f64_eddy", 600.0, 3, physics="dcmip"),
        # the smallest call: one surface field analysed on the test-bed grid
        _transform("grdtospec_t42_1_fp64", "grdtospec", 42, 128, 64, 1, "fp64", False),
        # winds of one 64-level history record for post-processing, single precision
        _transform("getuv_t254_64_single", "getuv", 254, 768, 384, 64, "tf32x3", True),
        # vorticity and divergence of 64 levels of analysed winds, double precision
        _transform("getvrtdivspec_t126_64_fp64", "getvrtdivspec", 126, 384, 190, 64, "fp64", False),
        # one training minibatch of the closure driver
        _closure("closure_grad_4096", "loss_grad", 64, 256, 3, 4096),
        # closure inference over the columns of the 192 x 94 grid
        _closure("closure_forward_18048", "forward", 64, 256, 3, 18048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(T, rng):
    """The quadratic Gaussian grid of a truncation: nlon the next even 2^a 3^b above 3 T, about half as many rows."""
    nlon = 3 * T + 1
    while True:
        n = nlon
        while n % 2 == 0:
            n //= 2
        while n % 3 == 0:
            n //= 3
        if n == 1 and nlon % 2 == 0:
            break
        nlon += 1
    return nlon, 2 * (nlon // 4) - rng.choice([0, 0, 2])


def draw(rng):
    kind = rng.choice(["forecast"] * 5 + ["transform"] * 3 + ["closure"] * 2)
    if kind == "forecast":
        prec = rng.choice(["fp64", "fp64", "tf32x3", "tf32x3", "tf32x3", "f64_eddy", "f64_tf32x3", "fp32"])
        T = _log_int(rng, 21, 126 if prec == "fp64" else 500 if prec == "tf32x3" else 192)
        nlon, nlat = _grid(T, rng)
        L = _log_int(rng, 10, 72)
        dt = 1200.0 if T <= 62 else 600.0 if T <= 126 else 300.0 if T <= 254 else 150.0
        physics = "dcmip" if prec in ("f64_eddy", "fp64") and rng.random() < 0.3 else "hs"
        steps = 1 if prec in ("tf32x3", "fp32") else rng.randint(2, 4)
        c = _forecast("", T, nlon, nlat, L, 3 if physics == "dcmip" else rng.randint(0, 4), prec, dt, steps, physics)
    elif kind == "transform":
        T = _log_int(rng, 21, 254)
        nlon, nlat = _grid(T, rng)
        prec = rng.choice(["fp64", "tf32x3", "tf32x3"])
        op = rng.choice(["spectogrd", "grdtospec", "getuv", "getvrtdivspec", "getgrad"])
        c = _transform("", op, T, nlon, nlat, _log_int(rng, 1, 96), prec, prec == "tf32x3" and rng.random() < 0.7)
    else:
        c = _closure("", rng.choice(["loss_grad", "forward"]), _log_int(rng, 10, 64), rng.choice([64, 96, 128, 192, 256]),
                     rng.randint(1, 4), _log_int(rng, 200, 18432))
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs --
_PHYS = dict(a=float(np.float32(6.3712e6)), rd=float(np.float32(287.05)), cp=float(np.float32(1004.6)),
             cvap=float(np.float32(1846.0)), omega=float(np.float32(7.2921e-5)))


def _vertical(L, eta_c=0.2, p0=1.0e5):
    """Hybrid coordinate, interfaces top to bottom: thin layers at both ends, pure pressure above eta_c."""
    eta = 0.5 * (1.0 - np.cos(np.pi * np.arange(L + 1) / L))
    bk = np.where(eta > eta_c, ((eta - eta_c) / (1.0 - eta_c)) ** 2, 0.0)
    ak = p0 * (eta - bk)
    ak[0] = bk[0] = ak[-1] = 0.0
    bk[-1] = 1.0
    return ak, bk, eta


def _degrees(T, device):
    order = np.repeat(np.arange(T + 1), T + 1 - np.arange(T + 1))
    deg = np.arange(order.size) - np.concatenate([[0], np.cumsum(T + 1 - np.arange(T + 1))])[order] + order
    return torch.from_numpy(deg).to(device), torch.from_numpy(order).to(device)


def _eddies(gen, T, nb, slope, rms, deg, order):
    """nb seeded fields of grid RMS rms with amplitudes n^slope, n >= 1 (complex128 [nb, nlm])."""
    z = torch.randn(nb, deg.numel(), 2, dtype=torch.float64, device=deg.device, generator=gen)
    z[:, order == 0, 1] = 0.0
    amp = torch.where(deg > 0, deg.clamp(min=1).double() ** slope, torch.zeros((), dtype=torch.float64, device=deg.device))
    z *= amp[:, None]
    w = torch.where(order == 0, 1.0, 2.0).to(torch.float64)
    ms = (z.square().sum(2) * w).sum(1) / (4 * math.pi)
    z *= (rms / ms.sqrt())[:, None, None]
    return torch.view_as_complex(z)


def _generator(seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.Generator(device=dev).manual_seed(seed), dev


def _model_state(c, seed):
    """vrt, div, tv, trc, lnps (levels bottom to top) in the host precision of the case."""
    gen, dev = _generator(seed)
    T, L, nt = c["T"], c["L"], c["nt"]
    deg, order = _degrees(T, dev)
    _, _, eta = _vertical(L)
    mid = torch.from_numpy(0.5 * (eta[1:] + eta[:-1])[::-1].copy()).to(dev)  # bottom to top
    y00 = math.sqrt(4 * math.pi)
    # eight vertical modes of falling weight: neighbouring levels are correlated, as they are in an atmosphere
    k = torch.arange(8, dtype=torch.float64, device=dev)
    modes = torch.cos(math.pi * (torch.arange(L, dtype=torch.float64, device=dev)[:, None] + 0.5) / L * k) / (1.0 + k)
    modes = (modes / modes.square().sum(1, keepdim=True).sqrt()).to(torch.complex128)

    def field(slope, rms):
        return modes @ _eddies(gen, T, 8, slope, rms, deg, order)

    st = dict(vrt=field(-2.0 / 3.0, 1.5e-5), div=field(-1.0 / 3.0, 1.0e-5), tv=field(-2.0, 4.0),
              lnps=_eddies(gen, T, 1, -2.0, 0.01, deg, order)[0])
    # the column's mass convergence is small beside the divergence of its levels
    mass = torch.from_numpy((eta[1:] - eta[:-1])[::-1].copy()).to(dev).to(torch.complex128)
    st["div"] -= 0.99 * (mass @ st["div"])
    st["tv"][:, 0] += (300.0 * mid ** 0.19).clamp(min=210.0) * y00
    st["lnps"][0] += math.log(1.0e5) * y00
    trc = []
    for q in range(nt):
        mean = 0.014 * mid ** 3 if c["physics"] == "dcmip" and q == 0 else torch.full_like(mid, 1.0e-3 * (q + 1))
        e = field(-2.0, 1.0) * (0.1 * mean)[:, None]
        e[:, 0] += mean * y00
        trc.append(e)
    st["trc"] = torch.stack(trc) if trc else torch.zeros(0, L, deg.numel(), dtype=torch.complex128, device=dev)
    ct = torch.complex128 if c["prec"] == "fp64" else torch.complex64
    return {k: v.to(ct) for k, v in st.items()}


def _transform_inputs(c, seed):
    gen, dev = _generator(seed)
    T, nb = c["T"], c["nb"]
    if c["op"] in ("grdtospec", "getvrtdivspec"):  # grid fields as a model has them: a mean, waves and noise
        lam = torch.linspace(0, 2 * math.pi, c["nlon"] + 1, dtype=torch.float64, device=dev)[:-1]
        phi = torch.linspace(math.pi / 2, -math.pi / 2, c["nlat"], dtype=torch.float64, device=dev)[:, None]
        out = []
        for i in range(1 if c["op"] == "grdtospec" else 2):
            ph = torch.rand(nb, 4, dtype=torch.float64, device=dev, generator=gen) * 2 * math.pi
            g = torch.zeros(nb, c["nlat"], c["nlon"], dtype=torch.float64, device=dev)
            for k in range(4):
                g += 8.0 / (k + 1) * torch.cos(phi) ** (k + 2) * torch.cos((k + 1) * lam + 3 * phi + ph[:, k, None, None])
            g += torch.cos(phi) * torch.randn(g.shape, dtype=torch.float64, device=dev, generator=gen)
            out.append(g + (280.0 if c["op"] == "grdtospec" else 0.0))
        t = torch.float32 if c["single"] else torch.float64
    else:
        deg, order = _degrees(T, dev)
        rms, slope = {"getuv": (1.0e-5, -1.0), "spectogrd": (5.0, -1.5), "getgrad": (5.0, -2.0)}[c["op"]]
        out = [_eddies(gen, T, nb, slope, rms, deg, order) for _ in range(2 if c["op"] == "getuv" else 1)]
        t = torch.complex64 if c["single"] else torch.complex128
    return [x.to(t) for x in out]


def _closure_inputs(c, seed):
    """Columns and targets of unit variance, and the packed parameters (He initialisation)."""
    gen, dev = _generator(seed)
    sizes = [3 * c["L"] + 1] + [c["hidden"]] * c["layers"] + [3 * c["L"]]
    shapes = [(sizes[i + 1], sizes[i]) for i in range(len(sizes) - 1)]
    rnd = lambda *s: torch.randn(*s, device=dev, generator=gen, dtype=torch.float32)  # noqa: E731
    layers = [(rnd(fo, fi) * math.sqrt(2.0 / fi), 0.05 * rnd(fo)) for fo, fi in shapes]
    return rnd(c["cols"], sizes[0]), rnd(c["cols"], sizes[-1]), layers


# ------------------------------------------------------------ prepare, run --
def _host(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    p.copy_(t)
    return p


def prepare(c, seed):
    if c["kind"] == "forecast":
        ak, bk, _ = _vertical(c["L"])
        kw = dict(dcmip=43, dry=False, heldsuarez=False) if c["physics"] == "dcmip" else {}
        model = core.Dycore(c["T"], c["nlon"], c["nlat"], c["L"], ak, bk, ntrac=c["nt"], dt=c["dt"], precision=c["prec"], **kw)
        st = {k: _host(v) for k, v in _model_state(c, seed).items()}
        out = {k: torch.empty_like(v, pin_memory=v.is_pinned()) for k, v in st.items()}
        for v in out.values():
            v.zero_()
        return dict(case=c, model=model, keep=(st, out), inp={k: v.numpy() for k, v in st.items()}, out={k: v.numpy() for k, v in out.items()})
    if c["kind"] == "transform":
        ak, bk, _ = _vertical(min(64, max(4, c["nb"])))
        model = core.Dycore(c["T"], c["nlon"], c["nlat"], len(ak) - 1, ak, bk, precision=c["prec"])
        return dict(case=c, model=model, inp=[x.cpu().numpy() for x in _transform_inputs(c, seed)])
    x, t, layers = _closure_inputs(c, seed)
    net = core.Mlp(x.shape[1], c["hidden"], c["layers"], t.shape[1], seed=1)
    net.set_params(np.concatenate([np.concatenate([w.cpu().numpy().ravel(), b.cpu().numpy()]) for w, b in layers]))
    return dict(case=c, net=net, x=x, t=t)


def run(s):
    c = s["case"]
    if c["kind"] == "forecast":
        g, i, o = s["model"], s["inp"], s["out"]
        g.set_state(i["vrt"], i["div"], i["tv"], i["lnps"], trc=i["trc"] if c["nt"] else None)
        g.advance(c["steps"])
        lib = core.load()
        get = lib.gd_get_state if o["vrt"].dtype == np.complex128 else lib.gd_get_state_f
        if get(g.h, *[o[k].ctypes.data_as(core.ctypes.c_void_p) if o[k].size else None for k in ("vrt", "div", "tv", "trc", "lnps")]) != core.GD_OK:
            raise RuntimeError(lib.gd_last_error(g.h).decode())
        return o
    if c["kind"] == "transform":
        return getattr(s["model"], c["op"])(*s["inp"])
    if c["op"] == "forward":
        return s["net"].forward(s["x"])
    return s["net"].loss_grad(s["x"], s["t"])


# ------------------------------------------------------------------- work --
def work(c):
    if c["kind"] == "closure":
        sizes = [3 * c["L"] + 1] + [c["hidden"]] * c["layers"] + [3 * c["L"]]
        w = sum(a * b for a, b in zip(sizes, sizes[1:]))
        n = c["cols"]
        if c["op"] == "forward":
            return dict(bytes=4.0 * n * (sizes[0] + sizes[-1]) + 2.0 * w, flops=2.0 * w * n)
        return dict(bytes=4.0 * n * (sizes[0] + sizes[-1]) + 6.0 * w, flops=2.0 * w * n + 2.0 * w * n + 2.0 * (w - sizes[0] * sizes[1]) * n)
    T, nlon, nlat = c["T"], c["nlon"], c["nlat"]
    nlm, ng, M = (T + 1) * (T + 2) // 2, nlon * nlat, nlon // 2
    leg = 2.0 * nlm * nlat  # one complex column through one table, hemispheres shared
    fft = nlat * (5.0 * M * math.log2(M) + 8.0 * M)  # one grid field
    if c["kind"] == "transform":
        nb = c["nb"]
        r = 4 if c["single"] else 8
        cols, fields, spec = {"spectogrd": (1, 1, 1), "grdtospec": (1, 1, 1), "getuv": (4, 2, 2), "getvrtdivspec": (4, 2, 2), "getgrad": (2, 2, 1)}[c["op"]]
        return dict(bytes=float(r * nb * (fields * ng + spec * 2 * nlm)), flops=nb * (cols * leg + fields * fft))
    L, nt = c["L"], c["nt"]
    r = 8 if c["prec"] == "fp64" else 4
    # columns through a Legendre table and grid fields through the longitude transform: three tendency
    # evaluations, then the physics' inverse and its increments
    cols = 3 * ((5 + nt) * L + 1 + (3 + nt) * L + 1 + (4 + nt) * L + 1 + 2 * L) + (5 + nt) * L + 2 * L + 2 + 3 * L + 1
    rows = 3 * ((7 + 3 * nt) * L + 3 + (4 + nt) * L + 1) + (5 + nt) * L + 3 + 3 * L + 1
    state = 2 * r * nlm * ((3 + nt) * L + 1)
    return dict(bytes=2.0 * state, flops=c["steps"] * (cols * leg + rows * fft))


# --------------------------------------------- 64-bit statement, plain torch --
class _Sphere:
    """Spherical-harmonic transforms in FP64: orthonormal harmonics without the Condon-Shortley phase, m-major
    triangular order, the m > 0 coefficients standing for the (+m, -m) pair."""

    def __init__(self, T, nlon, nlat, dev):
        self.T, self.nlon, self.nlat = T, nlon, nlat
        self.deg, self.order = _degrees(T, dev)
        self.a = _PHYS["a"]
        mu = np.cos(np.pi * (np.arange(nlat) + 0.75) / (nlat + 0.5))
        for _ in range(8):  # Newton on P_nlat
            p0, p1 = np.ones(nlat), mu.copy()
            for n in range(2, nlat + 1):
                p0, p1 = p1, ((2 * n - 1) * mu * p1 - (n - 1) * p0) / n
            d = nlat * (mu * p1 - p0) / (mu * mu - 1)
            mu = mu - p1 / d
        p0, p1 = np.ones(nlat), mu.copy()
        for n in range(2, nlat + 1):
            p0, p1 = p1, ((2 * n - 1) * mu * p1 - (n - 1) * p0) / n
        d = nlat * (mu * p1 - p0) / (mu * mu - 1)
        w = 2.0 / ((1 - mu * mu) * d * d)
        self.w = torch.from_numpy(w).to(dev)
        self.mu = torch.from_numpy(mu).to(dev)
        self.lat = torch.asin(self.mu)
        self.cos = torch.sqrt((1 - self.mu) * (1 + self.mu))
        self.off = [0]
        self.P, self.H = [], []
        # P_n^m for all m at once, by degree offset k = n - m
        m = torch.arange(T + 1, dtype=torch.float64, device=dev)
        fac = torch.cumsum(torch.cat([torch.zeros(1, dtype=torch.float64, device=dev), 0.5 * torch.log((2 * m[1:] + 1) / (2 * m[1:]))]), 0)
        pmm = torch.exp(fac[:, None] + m[:, None] * torch.log(self.cos)[None, :]) / math.sqrt(4 * math.pi)
        rows, prev, cur = [], torch.zeros_like(pmm), pmm
        for k in range(T + 1):
            keep = T + 1 - k  # orders with n = m + k <= T
            n = m[:keep] + k
            if k > 0:
                al = torch.sqrt((4 * n * n - 1) / (n * n - m[:keep] ** 2))
                be = torch.sqrt(((n - 1) ** 2 - m[:keep] ** 2) / (4 * (n - 1) ** 2 - 1))
                cur, prev = al[:, None] * (self.mu * cur[:keep] - be[:, None] * prev[:keep]), cur[:keep]
            rows.append(cur)
        for mm in range(T + 1):
            P = torch.stack([rows[k][mm] for k in range(T + 1 - mm)])
            n = torch.arange(mm, T + 1, dtype=torch.float64, device=dev)[:, None]
            c = torch.sqrt((n * n - mm * mm) * (2 * n + 1) / (2 * n - 1).clamp(min=1))
            below = torch.cat([torch.zeros_like(P[:1]), P[:-1]])
            self.P.append(P)
            self.H.append((-n * self.mu * P + c * below) / self.cos)
            self.off.append(self.off[-1] + T + 1 - mm)

    def fourier(self, tab, s):
        """[nb, nlm] -> [nb, T+1, nlat]"""
        out = torch.zeros(s.shape[0], self.T + 1, self.nlat, dtype=torch.complex128, device=s.device)
        for m in range(self.T + 1):
            x = s[:, self.off[m]:self.off[m + 1]]
            y = torch.cat([x.real, x.imag]) @ tab[m]
            out[:, m] = torch.complex(y[:s.shape[0]], y[s.shape[0]:])
        return out

    def grid(self, F):
        return torch.fft.irfft(F.transpose(1, 2), n=self.nlon, dim=2, norm="forward")

    def ungrid(self, g):
        return (torch.fft.rfft(g, dim=2, norm="forward")[:, :, :self.T + 1]).transpose(1, 2)

    def legendre(self, tab, F):
        F = F * (2 * math.pi * self.w)
        nb = F.shape[0]
        return torch.cat([torch.complex(*(torch.cat([F[:, m].real, F[:, m].imag]) @ tab[m].T).split(nb)) for m in range(self.T + 1)], 1)

    def im(self, F):
        return F * (1j * torch.arange(self.T + 1, dtype=torch.float64, device=F.device)[:, None] / self.cos)

    def spectogrd(self, s):
        return self.grid(self.fourier(self.P, s))

    def grdtospec(self, g):
        return self.legendre(self.P, self.ungrid(g))

    def invlap(self, s):
        lap = -self.deg.double() * (self.deg + 1)
        return torch.where(self.deg > 0, s / lap.clamp(max=-1.0), torch.zeros((), dtype=s.dtype, device=s.device))

    def getuv(self, vrt, div):
        s, x = self.a * self.invlap(vrt), self.a * self.invlap(div)
        u = self.im(self.fourier(self.P, x)) - self.fourier(self.H, s)
        v = self.im(self.fourier(self.P, s)) + self.fourier(self.H, x)
        return self.grid(u), self.grid(v)

    def getvrtdivspec(self, u, v):
        U, V = self.ungrid(u), self.ungrid(v)
        vrt = (self.legendre(self.P, self.im(V)) + self.legendre(self.H, U)) / self.a
        return vrt, (self.legendre(self.P, self.im(U)) - self.legendre(self.H, V)) / self.a

    def getgrad(self, s):
        return self.grid(self.im(self.fourier(self.P, s))) / self.a, self.grid(self.fourier(self.H, s)) / self.a


def _f32(x):
    return float(np.float32(x))


class _Model:
    """The Held-Suarez step in FP64: hydrostatic tendencies on hybrid levels, the IMEX RK3 scheme with the
    per-degree semi-implicit solve, hyperdiffusion, the forcing and the dry-mass fixer.  3-D fields are
    [level bottom to top], interface quantities top to bottom."""

    def __init__(self, c, dev):
        self.c, self.dev = c, dev
        L, T, dt = c["L"], c["T"], c["dt"]
        S = self.S = _Sphere(T, c["nlon"], c["nlat"], dev)
        ak, bk, _ = _vertical(L)
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)  # noqa: E731
        self.rd, self.cp, self.a = _PHYS["rd"], _PHYS["cp"], _PHYS["a"]
        self.kappa = self.rd / self.cp
        self.ak, self.bk = t(ak), t(bk)
        self.dbk, self.ck = t(bk[1:] - bk[:-1]), t(ak[1:] * bk[:-1] - ak[:-1] * bk[1:])
        self.lap = -S.deg.double() * (S.deg + 1)
        # damping profiles
        si = (ak / 101300.0 + bk)[::-1]
        sl = 0.5 * (si[1:] + si[:-1])
        if T > 170:
            x4 = np.float32(np.float32(T) / np.float32(170)) ** 2
            efold, fshk = 3600.0 / (float(np.float32(x4 * x4)) * _f32(1.1)), _f32(2.2)
        else:
            efold = 1.0 / (_f32(12.0e15 if T in (126, 170) else 3.0e15) / self.a ** 4 * 41990400.0)
            fshk = _f32(1.5) if T == 126 else 1.0
        efold *= 2.0
        self.dp = t(sl ** math.log(1.0 / fshk))
        self.mp = t(np.where(sl < _f32(0.002), np.log(_f32(0.002) / sl) / (5.0 * 86400.0), 0.0))
        self.dis = -(1.0 / efold) * (self.lap / self.lap.min()) ** 4
        # linear gravity-wave operators about an isothermal 300 K state at 800 hPa
        pk = ak + bk * 800.0e2
        dpk = pk[1:] - pk[:-1]
        ln = np.concatenate([[0.0], np.log(pk[2:] / pk[1:-1])])
        alfa = np.concatenate([[_f32(np.log(np.float32(2.0)))], 1.0 - pk[1:-1] / dpk[1:] * ln[1:]])
        ye, te = np.zeros((L, L)), np.zeros((L, L))
        for i in range(L):
            ye[i, i], te[i, i] = alfa[i] * self.rd, self.kappa * 300.0 * alfa[i]
            ye[i, i + 1:] = self.rd * ln[i + 1:]
            te[i, :i] = self.kappa * 300.0 * dpk[:i] / dpk[i] * ln[i]
        self.A, self.B = t(ye[::-1, ::-1] / self.a ** 2), t(te[::-1, ::-1])
        self.sv = t((dpk / 800.0e2)[::-1])
        self.tor = torch.full((L,), self.rd * 300.0 / self.a ** 2, dtype=torch.float64, device=dev)
        ym = torch.outer(self.tor, self.sv) + self.A @ self.B
        nn = torch.arange(T + 1, dtype=torch.float64, device=dev)
        eye = torch.eye(L, dtype=torch.float64, device=dev)
        self.D = [torch.linalg.inv(eye + ((f * dt) ** 2 * nn * (nn + 1))[:, None, None] * ym) for f in (_f32(1 / 6), _f32(1 / 3), 0.25)]
        self.by_degree = [torch.nonzero(S.deg == n)[:, 0] for n in range(T + 1)]

    def lnp(self, ps):
        """pk, dpk (layers), ln(p below / p above) and alfa, one layer from the top each"""
        pk = [self.ak[i] + self.bk[i] * ps for i in range(self.c["L"] + 1)]
        rl = [torch.full_like(ps, _f32(99999.99))] + [torch.log(pk[k + 1] / pk[k]) for k in range(1, self.c["L"])]
        return pk, rl

    def tend(self, s):
        S, L, nt = self.S, self.c["L"], self.c["nt"]
        u, v = S.getuv(s["vrt"], s["div"])
        zeta, div, tv = S.spectogrd(s["vrt"]), S.spectogrd(s["div"]), S.spectogrd(s["tv"])
        tx, ty = S.getgrad(s["tv"])
        lx, ly = (g[0] for g in S.getgrad(s["lnps"][None]))
        ps = torch.exp(S.spectogrd(s["lnps"][None])[0])
        if self.pdry is None:
            self.pdry = self.mean(ps)
        q = [S.spectogrd(x) for x in s["trc"]]
        pk, rl = self.lnp(ps)
        fcor = (2.0 * _PHYS["omega"] * torch.sin(S.lat))[:, None]
        dbs, cbs = [torch.zeros_like(ps)], [torch.zeros_like(ps)]  # sums over the layers above
        for k in range(L):
            b = L - 1 - k
            dbs.append(dbs[-1] + div[b] * (pk[k + 1] - pk[k]))
            cbs.append(cbs[-1] + (u[b] * lx + v[b] * ly) * self.dbk[k])
        dlnps = -dbs[L] / ps - cbs[L]
        eta = [torch.zeros_like(ps)] + [-ps * (self.bk[k] * dlnps + cbs[k]) - dbs[k] for k in range(1, L)] + [torch.zeros_like(ps)]
        fu, fv, dtv, ke = (torch.empty_like(u) for _ in range(4))
        dq = [torch.empty_like(x) for x in q]
        below = [torch.zeros_like(ps) for _ in range(3)]  # pressure-gradient sums over the layers below
        half = [self.halves(x, eta) for x in q]
        for b in range(L):
            k = L - 1 - b
            dp, cg = pk[k + 1] - pk[k], u[b] * lx + v[b] * ly
            al = torch.full_like(ps, _f32(np.log(np.float32(2.0)))) if k == 0 else 1.0 - pk[k] / dp * rl[k]
            if k == 0:
                wb = al * (div[b] * dp + ps * cbs[1] * self.dbk[0])
                wc = ps * cg * self.dbk[0]
            else:
                wb = rl[k] * (dbs[k] + ps * cbs[k]) + al * (div[b] * dp + ps * cg * self.dbk[k])
                wc = ps * cg * (self.dbk[k] + self.ck[k] * rl[k] / dp)
            om = (wc - wb) / dp
            cofb1 = -(al * self.dbk[k]) / dp if k == 0 else -(self.bk[k] * rl[k] + al * self.dbk[k]) / dp
            cofa = -(self.bk[k + 1] * pk[k] / pk[k + 1] - self.bk[k] + rl[k] * (self.bk[k] - pk[k] * self.dbk[k] / dp)) / dp
            common = (cofb1 - cofa) * self.rd * tv[b] * ps - self.rd * below[0] * ps
            gx = common * lx - self.rd * (below[1] + al * tx[b])
            gy = common * ly - self.rd * (below[2] + al * ty[b])

            def vadv(f):
                acc = torch.zeros_like(ps)
                if b > 0:
                    acc = acc + eta[k + 1] * (f[b - 1] - f[b])
                if b + 1 < L:
                    acc = acc + eta[k] * (f[b] - f[b + 1])
                return 0.5 / dp * acc

            heat = self.kappa * om * tv[b]
            if nt:
                heat = heat / (1.0 + (_PHYS["cvap"] / self.cp - 1.0) * q[0][b])
            dtv[b] = -u[b] * tx[b] - v[b] * ty[b] - vadv(tv) + heat
            fu[b] = u[b] * (zeta[b] + fcor) + vadv(v) - gy
            fv[b] = v[b] * (zeta[b] + fcor) - vadv(u) + gx
            ke[b] = 0.5 * (u[b] ** 2 + v[b] ** 2)
            for i in range(nt):
                h = half[i]
                dq[i][b] = -(h[k + 1] * eta[k + 1] - h[k] * eta[k] + q[i][b] * (eta[k] - eta[k + 1])) / dp
            if k > 0:
                below[0] = below[0] + (self.bk[k + 1] / pk[k + 1] - self.bk[k] / pk[k]) * tv[b]
                below[1] = below[1] + rl[k] * tx[b]
                below[2] = below[2] + rl[k] * ty[b]
        for i in range(nt):
            qx, qy = S.getgrad(s["trc"][i])
            dq[i] -= u * qx + v * qy
        ddiv, mdvrt = S.getvrtdivspec(fu, fv)
        return dict(vrt=-mdvrt, div=ddiv - self.lap / self.a ** 2 * S.grdtospec(ke), tv=S.grdtospec(dtv),
                    trc=torch.stack([S.grdtospec(x) for x in dq]) if nt else torch.zeros_like(s["trc"]), lnps=S.grdtospec(dlnps[None])[0])

    def halves(self, q, eta):
        """Thuburn-limited tracer at the interfaces, top to bottom"""
        L, tiny = self.c["L"], np.finfo(np.float64).tiny
        top, bot = q[L - 1], q[0]
        d = [None] * (L + 1)
        two = 2.0 * top - q[L - 2]
        d[0] = torch.where(top >= 0, top - two.clamp(min=0.0), top - two.clamp(max=0.0))
        two = 2.0 * bot - q[1]
        d[L] = torch.where(bot >= 0, two.clamp(min=0.0) - bot, two.clamp(max=0.0) - bot)
        for k in range(1, L):
            x = q[L - 1 - k] - q[L - k]
            d[k] = torch.where(x.abs() < tiny, torch.copysign(torch.full_like(x, tiny), x), x)
        h = [top]
        for k in range(1, L):
            up = eta[k] > 0.0
            r = torch.where(up, d[k - 1], d[k + 1]) / d[k]
            qu = torch.where(up, q[L - k], q[L - 1 - k])
            lim = torch.where(r > 0, 2.0 / (1.0 + 1.0 / r.clamp(min=tiny)), torch.zeros_like(r))
            h.append(qu + lim * (0.5 * (q[L - 1 - k] + q[L - k]) - qu))
        return h + [bot]

    def mean(self, f):
        return float((f * (self.S.w / (2.0 * self.c["nlon"]))[:, None]).sum())

    def rmul(self, M, x):
        return torch.complex(M @ x.real, M @ x.imag)

    def lin(self, s):
        return dict(div=-self.lap * (self.rmul(self.A, s["tv"]) + self.tor[:, None] * s["lnps"]), tv=-self.rmul(self.B, s["div"]),
                    lnps=-self.rmul(self.sv[None], s["div"])[0])

    def step(self, s):
        dt = self.c["dt"]
        ce = [[_f32(1 / 3)], [_f32(1 / 6), 0.5], [0.5, -0.5, 1.0]]
        ci = [[_f32(1 / 6)], [_f32(1 / 3), 0.0], [_f32(3 / 8), 0.0, _f32(3 / 8)]]
        imp = [_f32(1 / 6), _f32(1 / 3), 0.25]
        o, N, Z = s, [], []
        for r in range(3):
            t, l = self.tend(s), self.lin(s)
            for k in l:
                t[k] = t[k] - l[k]
            N.append(t)
            Z.append(l)
            s = {k: o[k] + dt * sum(e * n[k] for e, n in zip(ce[r], N)) for k in o}
            for k in Z[0]:
                s[k] = s[k] + dt * sum(e * z[k] for e, z in zip(ci[r], Z))
            rhs = s["div"] - imp[r] * dt * self.lap * (self.rmul(self.A, s["tv"]) + self.tor[:, None] * s["lnps"])
            div = torch.empty_like(rhs)
            for n, at in enumerate(self.by_degree):
                div[:, at] = self.rmul(self.D[r][n], rhs[:, at])
            s["div"] = div
            s["tv"] = s["tv"] - imp[r] * dt * self.rmul(self.B, div)
            s["lnps"] = s["lnps"] - imp[r] * dt * self.rmul(self.sv[None], div)[0]
        dd = self.dis * self.dp[:, None]
        s["vrt"], s["div"] = (s[k] / (1.0 - (dd - self.mp[:, None]) * dt) for k in ("vrt", "div"))
        s["tv"], s["trc"] = s["tv"] / (1.0 - dd * dt), s["trc"] / (1.0 - dd * dt)
        return self.physics(s)

    def physics(self, s):
        S, L, dt = self.S, self.c["L"], self.c["dt"]
        ps = torch.exp(S.spectogrd(s["lnps"][None])[0])
        sl, cl = torch.sin(S.lat)[:, None], torch.cos(S.lat)[:, None]
        pk, _ = self.lnp(ps)
        kf, ka, ks = (_f32(np.float32(1.0) / (np.float32(d) * np.float32(86400.0))) for d in (1.0, 40.0, 4.0))
        inc = {}
        for k in ("vrt", "div", "tv"):
            g = S.spectogrd(s[k])
            for b in range(L):
                lo, up = pk[L - b], pk[L - 1 - b]
                prs = ((lo ** self.kappa * lo - up ** self.kappa * up) / ((self.kappa + 1.0) * (lo - up))) ** (1.0 / self.kappa)
                bl = ((prs / ps - _f32(0.7)) / (1.0 - _f32(0.7))).clamp(min=0.0)
                if k == "tv":
                    teq = ((prs / 1.0e5) ** _f32(np.float32(2.0) / np.float32(7.0)) * (315.0 - 60.0 * sl ** 2 - 10.0 * torch.log(prs / 1.0e5) * cl ** 2)).clamp(min=200.0)
                    g[b] = (ka + (ks - ka) * bl * cl ** 4) * (teq - g[b])
                else:
                    g[b] = -(bl * kf) * g[b]
            inc[k] = S.grdtospec(g)
        s = {k: s[k] + dt * inc[k] if k in inc else s[k] for k in s}
        s["lnps"] = S.grdtospec(torch.log(ps * (self.pdry / self.mean(ps)))[None])[0]
        return s

    def run(self, s, steps):
        self.pdry = None
        for _ in range(steps):
            s = self.step(s)
        return s


def _exact_closure(c, seed):
    x, t, layers = _closure_inputs(c, seed)
    a, cache = x.double(), []
    layers = [(w.to(torch.bfloat16).double(), b.double()) for w, b in layers]  # weights are read in bfloat16
    for i, (w, b) in enumerate(layers):
        z = a @ w.T + b
        cache.append((a, z))
        a = z if i == len(layers) - 1 else 0.5 * z * (1.0 + torch.erf(z * math.sqrt(0.5)))
    if c["op"] == "forward":
        return a
    d = a - t.double()
    g, grads = 2.0 * d / d.numel(), []
    for i in range(len(layers) - 1, -1, -1):
        a, z = cache[i]
        if i < len(layers) - 1:
            g = g * (0.5 * (1.0 + torch.erf(z * math.sqrt(0.5))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi))
        grads[:0] = [(g.T @ a).reshape(-1), g.sum(0)]
        g = g @ layers[i][0]
    return float(d.square().mean()), torch.cat(grads).cpu().numpy()


def exact(c, seed):
    if c["kind"] == "closure":
        return _exact_closure(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "transform":
        x = [v.to(torch.complex128 if v.is_complex() else torch.float64) for v in _transform_inputs(c, seed)]
        y = getattr(_Sphere(c["T"], c["nlon"], c["nlat"], dev), c["op"])(*x)
        return tuple(v.cpu().numpy() for v in y) if isinstance(y, tuple) else y.cpu().numpy()
    # the moist physics has no plain statement here; the largest model would take minutes
    if c["physics"] != "hs" or c["T"] > 300:
        return None
    s = {k: v.to(torch.complex128) for k, v in _model_state(c, seed).items()}
    s = _Model(c, dev).run(s, c["steps"])
    return {k: s[k].cpu().numpy() for k in ("vrt", "div", "tv", "trc", "lnps")}
