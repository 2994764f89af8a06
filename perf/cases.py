"""The work that a user of this framework has it do, as cases that can be timed and compared.

Every case is one call through the public entry points (the C ABI of include/sfb_gpu.h by its Python
binding, as a pipeline with its catalogue on the device or in pinned host memory makes it):

* ``catalogue``        cat2amln of a galaxy catalogue on the device (sfb_cat2amln_device)
* ``mocks``            cat2amln of a batch of mock catalogues in pinned host memory (sfb_cat2amln_batched)
* ``field``            field2anlm of a shell x pixel field in pinned host memory (sfb_field2anlm_typed)
* ``synthesis``        anlm2field, the coefficients back to a field (sfb_anlm2field)
* ``field_gradient``   the gradient of a loss of field2anlm by the field (sfb_field2anlm_vjp_typed)
* ``weight_gradient``  the gradient of a loss of cat2amln by the galaxy weights (sfb_cat2amln_vjp)

``exact`` restates each of them in 64 bits with torch and numpy: HEALPix pixels, lambda_lm by its
recursion, ring FFTs, the Jacobi refinement in pixel space, one map per (n, l) pair and the g_nl cubic
splines (whose tables are an input of the call).
"""

import ctypes
import math
import os
import sys
from functools import lru_cache

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "sphericalfourierbesseldecompositions.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sfbgpu  # noqa: E402
from sfbgpu import _capi as capi  # noqa: E402
from sfbgpu.cat2anlm import GPUPlan  # noqa: E402

NITER = 3
# cos(theta) range of the survey footprints
SKY = {"full": (-1.0, 1.0), "cap": (0.5, 1.0), "band": (-0.3, 0.6)}


def listed():
    return [
        # the smallest call: a few thousand galaxies on a coarse grid (quick looks, unit tests, one of very
        # many light mocks); launches and latency count
        dict(name="catalogue_tiny", path="catalogue", precision="mixed", kmax=0.03, rmin=500.0, rmax=1000.0,
             nside=16, nr=100, ngal=5003, sky="cap", weights=True, window="separable"),
        # the reference's CPU-sized configuration: full sky, unit weights
        dict(name="catalogue_small", path="catalogue", precision="mixed", kmax=0.05, rmin=500.0, rmax=1000.0,
             nside=32, nr=250, ngal=200000, sky="full", weights=False, window="separable"),
        # a survey whose depth varies over the sky, so that its window does not separate: one window map per (n, l)
        dict(name="catalogue_dense", path="catalogue", precision="mixed", kmax=0.05, rmin=300.0, rmax=1300.0,
             nside=64, nr=150, ngal=300017, sky="cap", weights=True, window="dense"),
        # an ordinary survey: a million weighted galaxies in a band
        dict(name="catalogue_medium", path="catalogue", precision="mixed", kmax=0.06, rmin=500.0, rmax=1500.0,
             nside=128, nr=400, ngal=1234567, sky="band", weights=True, window="separable"),
        # the benchmark's workload: 1e7 galaxies in a 60 degree cap, nside 256
        dict(name="catalogue_large", path="catalogue", precision="mixed", kmax=0.1, rmin=500.0, rmax=2500.0,
             nside=256, nr=1000, ngal=10000000, sky="cap", weights=True, window="separable"),
        # all of it in FP64, the default precision of a plan
        dict(name="catalogue_fp64", path="catalogue", precision="fp64", kmax=0.06, rmin=500.0, rmax=1500.0,
             nside=128, nr=400, ngal=600011, sky="cap", weights=True, window="separable"),
        # mock catalogues for a covariance, one geometry and window, uneven sizes
        dict(name="mocks", path="mocks", precision="mixed", kmax=0.05, rmin=500.0, rmax=1000.0, nside=64, nr=250,
             ngal=200000, nmocks=8, sky="cap", weights=True, window="separable"),
        # a simulation's density shells in FP32 through the mixed transform
        dict(name="field_f32", path="field", precision="mixed", dtype="f32", kmax=0.06, rmin=500.0, rmax=1500.0,
             nside=128, nr=201),
        # the same direction in FP64
        dict(name="field_f64", path="field", precision="fp64", dtype="f64", kmax=0.05, rmin=300.0, rmax=1300.0,
             nside=64, nr=100),
        # coefficients back to a field
        dict(name="synthesis", path="synthesis", precision="fp64", kmax=0.06, rmin=500.0, rmax=1500.0, nside=128,
             nr=128),
        # field-level inference: the gradient by an FP32 field
        dict(name="field_gradient", path="field_gradient", precision="fp64", dtype="f32", kmax=0.06, rmin=500.0,
             rmax=1500.0, nside=128, nr=64),
        # the gradient by the galaxy weights
        dict(name="weight_gradient", path="weight_gradient", precision="fp64", kmax=0.05, rmin=300.0, rmax=1300.0,
             nside=64, nr=150, ngal=500009, sky="cap"),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    path = rng.choice(["catalogue", "catalogue", "catalogue", "catalogue", "mocks", "field", "field", "synthesis",
                       "field_gradient", "weight_gradient"])
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"]) if path in ("catalogue", "mocks", "field") else "fp64"
    top = 200.0 if (precision == "mixed" and path == "catalogue") else 90.0
    lk = _log(rng, 24.0, top)                           # kmax rmax, a little above lmax
    rmin = round(rng.uniform(200.0, 600.0), 1)
    rmax = round(rmin + _log(rng, 400.0, 1800.0), 1)
    kmax = round(lk / rmax, 5)
    nside = max(16, int(sfbgpu.estimate_nside(math.ceil(lk))) // rng.choice([1, 1, 2]))
    case = dict(path=path, precision=precision, kmax=kmax, rmin=rmin, rmax=rmax, nside=nside)
    if path in ("catalogue", "mocks", "weight_gradient"):
        case["sky"] = rng.choice(["full", "cap", "band"])
        case["nr"] = rng.randint(80, 500)
    if path == "catalogue":
        case["ngal"] = int(_log(rng, 3e3, 8e6 if precision == "mixed" else 1e6))
        case["weights"] = rng.random() < 0.7
        dense = lk < 60.0 and nside <= 64 and rng.random() < 0.25
        case["window"] = "dense" if dense else "separable"
    elif path == "mocks":
        case["ngal"] = int(_log(rng, 1e4, 1e6))
        case["nmocks"] = rng.randint(2, 9)
        case["weights"] = rng.random() < 0.7
        case["window"] = "separable"
    elif path == "weight_gradient":
        case["ngal"] = int(_log(rng, 3e3, 1e6))
    else:
        case["nr"] = int(_log(rng, 9, 201 if precision == "mixed" else 129 if path == "synthesis" else 65))
        if path != "synthesis":
            case["dtype"] = rng.choice(["f32", "f64"])
    return case


# --------------------------------------------------------------------------- what a program keeps
@lru_cache(maxsize=24)
def _amodes(kmax, rmin, rmax, nside):
    return sfbgpu.AnlmModes(kmax, rmin, rmax, nside=nside)


@lru_cache(maxsize=16)
def _plan(kmax, rmin, rmax, nside, precision):
    return GPUPlan(_amodes(kmax, rmin, rmax, nside), niter=NITER, precision=precision)


def _selection(r, rmin, rmax):
    return np.exp(-((r - (rmin + rmax) / 2) / (0.25 * (rmax - rmin))) ** 2 / 2)


def _depth(r, phi, rmin, rmax):
    """The part of the galaxies at r that a survey of uneven depth still sees at longitude phi."""
    return 1.0 - 0.5 * (r - rmin) / (rmax - rmin) * (0.5 + 0.5 * np.cos(phi))


@lru_cache(maxsize=16)
def _window(kmax, rmin, rmax, nside, nr, sky, kind):
    """(win_rhat_ln on the host, V_eff) of the survey's window on nr shells."""
    amodes = _amodes(kmax, rmin, rmax, nside)
    wm = sfbgpu.ConfigurationSpaceModes(rmin, rmax, nr, nside)
    th, ph = sfbgpu.pix2ang_ring(nside, np.arange(wm.npix))
    lo, hi = SKY[sky]
    z = np.cos(th)
    mask = ((z >= lo) & (z <= hi)).astype(float)
    phi = _selection(wm.r, rmin, rmax)
    from sfbgpu.cat2anlm import win_rhat_ln
    if kind == "separable":
        sep = sfbgpu.SeparableArray(phi, mask, "phi", "mask")
        return win_rhat_ln(sep, wm, amodes), sfbgpu.integrate_window(sep, wm)
    W = phi[:, None] * mask[None, :] * _depth(wm.r[:, None], ph[None, :], rmin, rmax)
    return win_rhat_ln(W, wm, amodes), sfbgpu.integrate_window(W, wm)


def _geometry(case):
    return case["kmax"], case["rmin"], case["rmax"], case["nside"]


def _catalogue(case, seed, ngal, dense=False):
    """(N, 3) r, theta, phi and weights on the device: r from r^2 times the radial selection, directions
    uniform in the footprint; thinned by the depth for a window that does not separate."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rmin, rmax = case["rmin"], case["rmax"]
    grid = np.linspace(rmin, rmax, 1 << 14)
    pdf = grid ** 2 * _selection(grid, rmin, rmax)
    cdf = np.concatenate([[0.0], np.cumsum(0.5 * (pdf[1:] + pdf[:-1]))])
    nq = 1 << 14
    rq = torch.from_numpy(np.interp(np.linspace(0.0, cdf[-1], nq + 1), cdf, grid)).cuda()
    n = int(1.7 * ngal) + 1000 if dense else ngal

    def u():
        return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)

    q = u() * nq
    j = q.long().clamp_(max=nq - 1)
    r = rq[j] + (q - j) * (rq[j + 1] - rq[j])
    lo, hi = SKY[case["sky"]]
    rtp = torch.stack([r, torch.arccos(lo + (hi - lo) * u()), 2 * math.pi * u()], dim=1)
    if dense:
        part = 1.0 - 0.5 * (rtp[:, 0] - rmin) / (rmax - rmin) * (0.5 + 0.5 * torch.cos(rtp[:, 2]))
        rtp = rtp[u() < part][:ngal]
        n = rtp.shape[0]
    w = 0.5 + u()
    return rtp.contiguous(), w.contiguous()


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out


def _dp(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def _vp(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _mock_sizes(case):
    n, k = case["ngal"], case["nmocks"]
    return [max(1, int(n * (0.3 + 1.4 * ((i * 5 + 2) % k) / k))) for i in range(k)]


def _normal(shape, seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=device, dtype=torch.float64)


def prepare(case, seed):
    plan = _plan(*_geometry(case), case["precision"])
    path = case["path"]
    s = {"path": path, "plan": plan, "rmin": case["rmin"], "rmax": case["rmax"]}
    if path in ("catalogue", "mocks"):
        win, veff = _window(*_geometry(case), case["nr"], case["sky"], case["window"])
        w = capi.Window()
        if case["window"] == "separable":
            mask = torch.from_numpy(np.ascontiguousarray(win.arr1))
            wln = torch.from_numpy(np.ascontiguousarray(win.arr2.T))       # Julia's (lmax+1) x nmax memory
            keep = [mask.cuda(), wln.cuda()] if path == "catalogue" else [_pinned(mask), _pinned(wln)]
            w.kind, w.mask, w.w_ln = capi.SFB_WINDOW_SEPARABLE, _dp(keep[0]), _dp(keep[1])
        else:
            keep = [torch.from_numpy(np.ascontiguousarray(win.T)).cuda()]
            w.kind, w.dense = capi.SFB_WINDOW_DENSE, _dp(keep[0])
        s.update(window=w, keep=keep)
    if path == "catalogue":
        rtp, wt = _catalogue(case, seed, case["ngal"], case["window"] == "dense")
        s.update(rtp=rtp, weight=wt if case["weights"] else None, nbar=rtp.shape[0] / veff,
                 out=torch.empty(2 * plan.nlmsize, dtype=torch.float64, device="cuda"))
    elif path == "mocks":
        sizes = _mock_sizes(case)
        cats = [_catalogue(case, seed * 101 + k, n) for k, n in enumerate(sizes)]
        s.update(rtp=_pinned(torch.cat([c for c, _ in cats])),
                 weight=_pinned(torch.cat([v for _, v in cats])) if case["weights"] else None,
                 offsets=np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64),
                 nbar=np.array([n / veff for n in sizes]),
                 out=torch.empty((len(sizes), 2 * plan.nlmsize), dtype=torch.float64, pin_memory=True))
    elif path == "field":
        f = _normal((plan.npix, case["nr"]), seed)                          # (nr, npix) in Julia's order
        s.update(nr=case["nr"], dtype=capi.SFB_F32 if case["dtype"] == "f32" else capi.SFB_F64,
                 field=_pinned(f.float() if case["dtype"] == "f32" else f),
                 out=torch.empty(2 * plan.nlmsize, dtype=torch.float64, pin_memory=True))
    elif path == "synthesis":
        s.update(nr=case["nr"], anlm=_pinned(_coefficients(case, seed)),
                 out=torch.empty((plan.npix, case["nr"]), dtype=torch.float64, pin_memory=True))
    elif path == "field_gradient":
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        s.update(nr=case["nr"], dtype=capi.SFB_F32 if case["dtype"] == "f32" else capi.SFB_F64,
                 abar=_pinned(_coefficients(case, seed)),
                 out=torch.empty((plan.npix, case["nr"]), dtype=dt, pin_memory=True))
    elif path == "weight_gradient":
        rtp, _ = _catalogue(case, seed, case["ngal"])
        s.update(rtp=_pinned(rtp), nbar=_nbar_of(case), abar=_pinned(_coefficients(case, seed)),
                 out=torch.empty(rtp.shape[0], dtype=torch.float64, pin_memory=True))
    return s


def _nbar_of(case):
    lo, hi = SKY[case["sky"]]
    vol = 2 * math.pi * (hi - lo) * (case["rmax"] ** 3 - case["rmin"] ** 3) / 3
    return case["ngal"] / vol


def _coefficients(case, seed):
    """Gaussian a_nlm, real at m = 0, interleaved (re, im)."""
    amodes = _amodes(*_geometry(case))
    a = _normal((sfbgpu.getnlmsize(amodes), 2), seed)
    m = np.concatenate([np.arange(l + 1) for _, l in amodes.pairs()])
    a[torch.from_numpy(np.nonzero(m == 0)[0]).cuda(), 1] = 0.0
    return a.reshape(-1)


def run(s):
    lib, plan, path = capi.lib, s["plan"].handle, s["path"]
    if path == "catalogue":
        capi.check(lib.sfb_cat2amln_device(plan, _vp(s["rtp"]), _vp(s["weight"]), s["rtp"].shape[0], s["nbar"],
                                           ctypes.byref(s["window"]), _vp(s["out"]),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    elif path == "mocks":
        capi.check(lib.sfb_cat2amln_batched(plan, _vp(s["rtp"]), _vp(s["weight"]), capi.ptr(s["offsets"]),
                                            len(s["nbar"]), capi.ptr(s["nbar"]), ctypes.byref(s["window"]),
                                            _vp(s["out"])))
    elif path == "field":
        capi.check(lib.sfb_field2anlm_typed(plan, _vp(s["field"]), s["dtype"], s["nr"], s["rmin"], s["rmax"],
                                            _vp(s["out"])))
    elif path == "synthesis":
        capi.check(lib.sfb_anlm2field(plan, _vp(s["anlm"]), s["nr"], s["rmin"], s["rmax"], _vp(s["out"])))
    elif path == "field_gradient":
        capi.check(lib.sfb_field2anlm_vjp_typed(plan, _vp(s["abar"]), s["nr"], s["rmin"], s["rmax"], _vp(s["out"]),
                                                s["dtype"]))
    elif path == "weight_gradient":
        capi.check(lib.sfb_cat2amln_vjp(plan, _vp(s["rtp"]), s["rtp"].shape[0], s["nbar"], _vp(s["abar"]),
                                        _vp(s["out"])))
    return s["out"]


def work(case):
    """Inputs and outputs once; the spherical-harmonic transforms of as many maps as the radial functions
    need (two per radial mode for a catalogue, one per shell of a field), one analysis or synthesis and
    NITER refinements (a synthesis and an analysis each), 4 flop per ring, (l, m) and map."""
    lmax = 0.95 * case["kmax"] * case["rmax"]
    nmax = case["kmax"] * (case["rmax"] - case["rmin"]) / math.pi
    npix, rings, lm = 12 * case["nside"] ** 2, 4 * case["nside"] - 1, lmax * lmax / 2
    nlm = nmax * lm / 3
    path = case["path"]
    n = case.get("ngal", 0)
    esz = 4 if case.get("dtype") == "f32" else 8
    passes = 1 if path == "synthesis" else 1 + 2 * NITER
    if path == "catalogue" and case["window"] == "dense":
        maps, io = nmax * lmax / 2, 8 * n * 4 + 8 * npix * nmax * lmax / 2 + 16 * nlm
    elif path == "catalogue":
        maps, io = 2 * nmax, 8 * n * 4 + 8 * npix + 16 * nlm
    elif path == "mocks":
        k = case["nmocks"]
        maps, io = 2 * nmax * k, 8 * sum(_mock_sizes(case)) * 4 + 16 * nlm * k
    elif path == "weight_gradient":
        maps, io = 2 * nmax, 8 * n * 4 + 16 * nlm
    else:
        maps, io = case["nr"], case["nr"] * npix * (8 if path == "synthesis" else esz) + 16 * nlm
    return {"bytes": float(io), "flops": 4.0 * maps * rings * lm * passes}


# --------------------------------------------------------------------------- the same in plain 64-bit torch
def _rings(ns):
    i = np.arange(1, 4 * ns)
    j = np.minimum(i, 4 * ns - i)                                  # ring counted from the nearer pole
    polar = j < ns
    npix = 12 * ns * ns
    nph = np.where(polar, 4 * j, 4 * ns)
    start = np.concatenate([[0], np.cumsum(nph)[:-1]])
    omz = np.where(polar, j * j / (3.0 * ns * ns), 1.0)
    zeq = (2 * ns - i) * (2.0 / (3.0 * ns))                             # outside the belt unused
    z = np.where(polar, np.where(i < 2 * ns, 1.0 - omz, omz - 1.0), zeq)
    sth = np.where(polar, np.sqrt(omz * (2.0 - omz)), np.sqrt(np.abs(1.0 - zeq * zeq)))
    phi0 = np.where(polar, np.pi / np.maximum(4 * j, 1), np.where((i + ns) % 2 == 1, 0.0, np.pi / (4 * ns)))
    return dict(nph=nph, start=start, z=z, sth=sth, phi0=phi0, npix=npix)


def _lambda(lmax, z, sth):
    """lambda_lm of every ring, [m, l, ring], by the upward recursion in l for all m at once, each value a
    double times a power of two kept apart (sin^m theta underflows near the poles)."""
    L, R = lmax, len(z)
    mant, expo = np.empty((L + 1, R)), np.zeros((L + 1, R), np.int64)
    c, e = np.full(R, 1.0 / math.sqrt(4 * math.pi)), np.zeros(R, np.int64)
    for m in range(L + 1):
        if m:
            c, d = np.frexp(-c * sth * math.sqrt((2 * m + 1) / (2.0 * m)))
            e = e + d
        mant[m], expo[m] = c, e
    out = np.zeros((L + 1, L + 1, R))
    v, old = mant.copy(), np.zeros((L + 1, R))
    ms = np.arange(L + 1, dtype=float)
    out[0, 0] = np.ldexp(mant[0], np.clip(expo[0], -2000, 2000))
    for l in range(1, L + 1):
        m = ms[:l]
        a = np.sqrt((4.0 * l * l - 1) / (l * l - m * m))[:, None]
        b = np.sqrt(((l - 1.0) ** 2 - m * m) / max(4.0 * (l - 1) ** 2 - 1, 1.0))[:, None]
        new = a * (z * v[:l] - b * old[:l])
        big = np.where(np.abs(new) > 2.0 ** 300, -600, 0)
        old[:l] = np.ldexp(v[:l], big)
        v[:l] = np.ldexp(new, big)
        expo[:l] -= big
        out[:l + 1, l] = np.ldexp(v[:l + 1], np.clip(expo[:l + 1], -2000, 2000))
    return out


class _SHT:
    def __init__(self, ns, lmax, dev):
        self.L, self.ns, self.dev = lmax, ns, dev
        r = _rings(ns)
        self.r, self.npix, self.w = r, r["npix"], 4 * math.pi / r["npix"]
        self.lam = torch.from_numpy(_lambda(lmax, r["z"], r["sth"])).to(dev)
        m = np.arange(lmax + 1)
        den = np.where(r["phi0"] > 0, np.round(np.pi / np.where(r["phi0"] > 0, r["phi0"], 1.0)), 1).astype(np.int64)
        ang = np.where(r["phi0"][:, None] > 0, np.pi * (m[None, :] % (2 * den[:, None])) / den[:, None], 0.0)
        self.ph = torch.from_numpy(np.exp(1j * ang)).to(dev)                  # e^{i m phi0}, [ring, m]
        # equal rings next to each other go through one FFT
        self.groups, k, n = [], 0, len(r["nph"])
        while k < n:
            j = k
            while j < n and r["nph"][j] == r["nph"][k]:
                j += 1
            self.groups.append((k, j, int(r["nph"][k]), int(r["start"][k])))
            k = j
        self.m = torch.arange(lmax + 1, device=dev)

    def analysis(self, f):                                                     # [b, npix] -> [m, l, b]
        b = f.shape[0]
        F = torch.empty((self.L + 1, len(self.r["nph"]), b), dtype=torch.complex128, device=self.dev)
        for k, j, n, s in self.groups:
            c = torch.fft.fft(f[:, s:s + (j - k) * n].reshape(b, j - k, n), dim=2)
            F[:, k:j] = (c[:, :, self.m % n] * (self.w * self.ph[k:j].conj())).permute(2, 1, 0)
        return torch.view_as_complex(torch.bmm(self.lam, torch.view_as_real(F).reshape(self.L + 1, -1, 2 * b))
                                     .reshape(self.L + 1, self.L + 1, b, 2))

    def synthesis(self, a):                                                    # [m, l, b] -> [b, npix]
        b = a.shape[2]
        G = torch.bmm(self.lam.transpose(1, 2), torch.view_as_real(a).reshape(self.L + 1, self.L + 1, 2 * b))
        G = torch.view_as_complex(G.reshape(self.L + 1, -1, b, 2))
        G[1:] *= 2
        G[0] = G[0].real + 0j
        f = torch.empty((b, self.npix), dtype=torch.float64, device=self.dev)
        for k, j, n, s in self.groups:
            c = torch.zeros((b, j - k, n), dtype=torch.complex128, device=self.dev)
            c.index_add_(2, self.m % n, (G[:, k:j].permute(2, 1, 0) * self.ph[k:j]).contiguous())
            f[:, s:s + (j - k) * n] = (torch.fft.ifft(c, dim=2) * n).real.reshape(b, -1)
        return f

    def map2alm(self, f):
        a = self.analysis(f)
        for _ in range(NITER):
            a = a + self.analysis(f - self.synthesis(a))
        return a

    def adjoint(self, abar):
        """The transpose of map2alm: w S sum_j (I - A S)^j E abar, E = 1/2 for m > 0."""
        e = abar.clone()
        e[1:] *= 0.5
        e[0] = e[0].real + 0j
        x = e
        for _ in range(NITER):
            x = e + x - self.analysis(self.synthesis(x))
        return self.w * self.synthesis(x)


def _pixel(ns, th, ph):
    """RING pixels (Gorski et al. 2005)."""
    npix = 12 * ns * ns
    z, t = torch.cos(th), torch.remainder(ph * (2.0 / math.pi), 4.0)
    t = torch.where(t >= 4.0, torch.zeros_like(t), t)
    za = z.abs()
    up, down = torch.floor(ns * (0.5 + t) - ns * z * 0.75).long(), torch.floor(ns * (0.5 + t) + ns * z * 0.75).long()
    ring = ns + 1 + up - down
    ip = ((up + down - ns + (1 - (ring & 1)) + 1 + 8 * ns) >> 1) % (4 * ns)
    belt = (2 * ns * (ns - 1) + (ring - 1) * 4 * ns + ip).clamp(0, npix - 1)
    tp, s = t - torch.floor(t), ns * torch.sqrt(3.0 * (1.0 - za))
    j = torch.floor(tp * s).long() + torch.floor((1.0 - tp) * s).long() + 1
    ip = torch.floor(t * j).long() % (4 * j)
    cap = torch.where(z > 0, 2 * j * (j - 1) + ip, npix - 2 * j * (j + 1) + ip)
    return torch.where(za <= 2.0 / 3.0, belt, cap)


def _spline(tab, r):
    x, y, ypp = (torch.from_numpy(np.ascontiguousarray(t)).to(r.device) for t in tab)
    h = (x[-1] - x[0]) / (len(x) - 1)
    i = ((r - x[0]) / h).long().clamp_(0, len(x) - 2)
    i = torch.where(r < x[i], i - 1, torch.where(r >= x[i + 1], i + 1, i)).clamp_(0, len(x) - 2)
    h = x[i + 1] - x[i]
    a, b = (x[i + 1] - r) / h, (r - x[i]) / h
    return a * y[i] + b * y[i + 1] + ((a ** 3 - a) * ypp[i] + (b ** 3 - b) * ypp[i + 1]) * (h * h / 6)


def _catalogue_exact(case, amodes, sht, rtp, w, nbar, win):
    pix = _pixel(case["nside"], rtp[:, 1], rtp[:, 2])
    scale = sht.npix / (4 * math.pi * nbar)
    pairs, out = amodes.pairs(), []
    for c in range(0, len(pairs), 128):
        chunk = pairs[c:c + 128]
        f = torch.zeros((len(chunk), sht.npix), dtype=torch.float64, device=sht.dev)
        for k, (n, l) in enumerate(chunk):
            v = _spline(amodes.basisfunctions.spline[(n, l)], rtp[:, 0])
            f[k].index_add_(0, pix, v if w is None else v * w)
            f[k] *= scale
            f[k] -= win(n, l)
        a = sht.map2alm(f)
        out += [a[:l + 1, l, k] for k, (n, l) in enumerate(chunk)]
    return torch.view_as_real(torch.cat(out)).reshape(-1)


def _shells(case, amodes, dev):
    rmin, rmax, nr = case["rmin"], case["rmax"], case["nr"]
    dr = (rmax - rmin) / nr
    r = torch.from_numpy(rmin + dr * (np.arange(nr) + 0.5)).to(dev)
    return r, dr, {p: _spline(amodes.basisfunctions.spline[p], r) for p in amodes.pairs()}


def _rows(amodes):
    at = 0
    for n, l in amodes.pairs():
        yield n, l, at
        at += l + 1


def _window_of(case, dev):
    win, veff = _window(*_geometry(case), case["nr"], case["sky"], case["window"])
    if case["window"] == "separable":
        mask = torch.from_numpy(win.arr1).to(dev)
        return (lambda n, l: mask * float(win.arr2[l, n - 1])), veff
    return (lambda n, l: torch.from_numpy(np.ascontiguousarray(win[:, l, n - 1])).to(dev)), veff


def exact(case, seed):
    dev = "cuda"
    amodes = _amodes(*_geometry(case))
    path, pairs, L = case["path"], amodes.pairs(), amodes.lmax
    npix, lm = 12 * case["nside"] ** 2, (L + 1) * (L + 1)
    per_pair = path in ("catalogue", "mocks", "weight_gradient")
    runs = case.get("nmocks", 1)
    maps = len(pairs) * runs if per_pair else case["nr"]
    # 8 flop per ring, (l, m) and map in every pass at about 0.6 TFLOP/s; 15 passes over each map's galaxies
    cost = maps * 4 * case["nside"] * lm * 8 * 7 / 6e11
    if per_pair:
        total = sum(_mock_sizes(case)) if path == "mocks" else case["ngal"]
        cost += len(pairs) * (total * 8 * 25 / 3e12 + runs * 3e-4)
    if cost > 12.0:
        return None
    sht = _SHT(case["nside"], L, dev)
    if path == "catalogue":
        rtp, w = _catalogue(case, seed, case["ngal"], case["window"] == "dense")
        win, veff = _window_of(case, dev)
        return _catalogue_exact(case, amodes, sht, rtp, w if case["weights"] else None, rtp.shape[0] / veff, win)
    if path == "mocks":
        win, veff = _window_of(case, dev)
        rows = []
        for k, n in enumerate(_mock_sizes(case)):
            rtp, w = _catalogue(case, seed * 101 + k, n)
            rows.append(_catalogue_exact(case, amodes, sht, rtp, w if case["weights"] else None, n / veff, win))
        return torch.stack(rows).cpu()
    if path == "weight_gradient":
        rtp, _ = _catalogue(case, seed, case["ngal"])
        ab = torch.view_as_complex(_coefficients(case, seed).reshape(-1, 2))
        pix = _pixel(case["nside"], rtp[:, 1], rtp[:, 2])
        out = torch.zeros(rtp.shape[0], dtype=torch.float64, device=dev)
        rows = list(_rows(amodes))
        for c in range(0, len(rows), 128):
            chunk = rows[c:c + 128]
            a = torch.zeros((L + 1, L + 1, len(chunk)), dtype=torch.complex128, device=dev)
            for k, (n, l, at) in enumerate(chunk):
                a[:l + 1, l, k] = ab[at:at + l + 1]
            f = sht.adjoint(a)
            for k, (n, l, at) in enumerate(chunk):
                out += _spline(amodes.basisfunctions.spline[(n, l)], rtp[:, 0]) * f[k][pix]
        return (out * (npix / (4 * math.pi * _nbar_of(case)))).cpu()
    r, dr, g = _shells(case, amodes, dev)
    if path == "field":
        f = _normal((npix, case["nr"]), seed)
        f = f.float().double() if case["dtype"] == "f32" else f
        a = sht.map2alm(f.T.contiguous())
        out = [(a[:l + 1, l] * (g[(n, l)] * r * r * dr)).sum(1) for n, l in pairs]
        return torch.view_as_real(torch.cat(out)).reshape(-1).cpu()
    ab = torch.view_as_complex(_coefficients(case, seed).reshape(-1, 2))
    a = torch.zeros((L + 1, L + 1, case["nr"]), dtype=torch.complex128, device=dev)
    for n, l, at in _rows(amodes):
        v = g[(n, l)] if path == "synthesis" else g[(n, l)] * r * r * dr
        a[:l + 1, l] += ab[at:at + l + 1, None] * v
    f = sht.synthesis(a) if path == "synthesis" else sht.adjoint(a)
    f = f.T.contiguous()
    return (f.float() if path == "field_gradient" and case["dtype"] == "f32" else f).cpu()
