"""GPU parity tests: libsfbgpu.so (through the C ABI) against the CPU oracle.

Tolerances (global relative error max|gpu - oracle| / max|oracle|):
* FP64 transforms and the spline radial mode: 1e-11 (same algorithm, FP64,
  only summation order differs);
* the piecewise-Legendre radial mode: 2e-7 against the reference algorithm
  (the expansion replaces the per-galaxy cubic spline; its projection error
  is reported by the plan and stays near the spline's own interpolation
  error).
"""

import numpy as np
import pytest

import sfbgpu
from sfbgpu import _capi as capi
from sfbgpu.cat2anlm import GPUPlan
from helpers import catalogue, modes_dict, record, rel_err, round_sig, ylm
from oracle import healpix as ohp, sfb as osfb, sht as osht

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    a = sfbgpu.AnlmModes(0.03, 500.0, 1000.0, nside=16)
    return a


# ---------------------------------------------------------------- HEALPix ----
def _near_boundaries(nside, rng, n=20_000):
    """Directions placed within +-1e-9 .. 1e-3 (in units of the floored
    quantities) of pixel edges: both edge families of the equatorial belt,
    the polar edges, |z| = 2/3 and quadrant edges of phi."""
    ns = float(nside)
    d = rng.choice([1e-9, -1e-9, 1e-6, -1e-6, 1e-4, -1e-4, 1e-3, -1e-3], n)
    out_th, out_ph = [], []
    # equatorial: ns (0.5 + tt) -+ 0.75 ns z = k + d
    z = rng.uniform(-0.66, 0.66, n)
    sgn = rng.choice([-1.0, 1.0], n)
    k = np.floor(ns * (0.5 + rng.uniform(0, 4, n)) - sgn * 0.75 * ns * z)
    tt = (k + d + sgn * 0.75 * ns * z) / ns - 0.5
    ok = (tt >= 0) & (tt < 4)
    out_th.append(np.arccos(z[ok]))
    out_ph.append(tt[ok] * np.pi / 2)
    # polar: tp * tmp = k + d (and (1 - tp) * tmp = k + d)
    za = rng.uniform(0.67, 0.9999, n)
    tmp = ns * np.sqrt(3 * (1 - za))
    k = np.floor(rng.uniform(0, 1, n) * tmp)
    tp = (k + d) / tmp
    tp = np.where(rng.random(n) < 0.5, tp, 1 - tp)
    ok = (tp > 0) & (tp < 1)
    q = rng.integers(0, 4, n)
    zz = np.where(rng.random(n) < 0.5, za, -za)
    out_th.append(np.arccos(zz[ok]))
    out_ph.append((q[ok] + tp[ok]) * np.pi / 2)
    # |z| = 2/3 and quadrant edges of phi
    out_th.append(np.arccos(np.array([2 / 3 + 1e-9, 2 / 3 - 1e-9, -2 / 3 + 1e-9, -2 / 3 - 1e-9, 2 / 3, -2 / 3])))
    out_ph.append(np.array([0.1, 1.0, 2.0, 3.0, 4.0, 5.0]))
    e = rng.uniform(0.1, 3.0, 400)
    out_th.append(e)
    out_ph.append(np.repeat([np.pi / 2, np.pi, 3 * np.pi / 2, 2 * np.pi], 100) + np.tile([1e-12, -1e-12, 1e-7, -1e-7], 100))
    return np.concatenate(out_th), np.concatenate(out_ph)


@pytest.mark.parametrize("nside", [1, 2, 7, 32, 256, 1024])
def test_ang2pix_bit_exact(nside):
    rng = np.random.default_rng(nside)
    n = 200_000
    th = np.arccos(rng.uniform(-1, 1, n))
    ph = rng.uniform(-2 * np.pi, 4 * np.pi, n)
    # pixel centres, poles, equator, phi edges (inputs whose cosine is exact in
    # every libm, so the pixel is determined by the ang2pix arithmetic alone)
    cth, cph = ohp.pix2ang_ring(nside, np.arange(min(12 * nside * nside, 50_000)))
    edge_th = np.array([0.0, np.pi, np.pi / 2, 1e-12, np.pi - 1e-12, 0.0, np.pi / 2])
    edge_ph = np.array([0.0, 2 * np.pi, -1e-15, np.pi / 2, 2 * np.pi - 1e-15, 1e300, -7.0])
    bth, bph = _near_boundaries(nside, rng)
    th = np.concatenate([th, cth, edge_th, bth])
    ph = np.concatenate([ph, cph, edge_ph, bph])
    gpu = sfbgpu.ang2pix_ring(nside, th, ph)
    ref = ohp.ang2pix_ring(nside, th, ph)
    assert np.all((gpu >= 0) & (gpu < 12 * nside * nside))
    assert np.array_equal(gpu, ref), f"{np.sum(gpu != ref)} mismatches"


# ---------------------------------------------------------------- SHT --------
@pytest.mark.parametrize("nside,lmax,niter", [(8, 23, 0), (8, 23, 3), (16, 31, 3), (16, 47, 3), (5, 14, 2)])
def test_map2alm_vs_oracle(nside, lmax, niter):
    a = sfbgpu.AnlmModes.from_nmax_lmax(1, lmax, 500.0, 1000.0, nside=nside, cache=True)
    plan = GPUPlan(a, niter=niter, radial="spline")
    rng = np.random.default_rng(lmax)
    maps = rng.normal(size=(3, 12 * nside * nside)) + 2.0
    out = sfbgpu.cat2anlm.map2alm(maps, a, niter=niter, radial="spline")
    S = osht.SHT(nside, lmax)
    ref = S.map2alm(maps, niter=niter)
    L = lmax
    tri = np.array([ref[b, l, m] for b in range(3) for l in range(L + 1) for m in range(l + 1)]).reshape(3, -1)
    record(f"map2alm_nside{nside}_lmax{lmax}_niter{niter}", rel_err(out, tri))
    assert rel_err(out, tri) < 1e-12
    plan.close()


@pytest.mark.parametrize("nmaps", [1, 2, 4])
def test_map2alm_few_maps_vs_oracle(nmaps):
    """One, two and four maps take the matrix-vector Legendre kernels."""
    nside, lmax = 16, 40
    a = sfbgpu.AnlmModes.from_nmax_lmax(1, lmax, 500.0, 1000.0, nside=nside, cache=True)
    rng = np.random.default_rng(nmaps)
    maps = rng.normal(size=(nmaps, 12 * nside * nside)) + 2.0
    out = sfbgpu.cat2anlm.map2alm(maps, a, niter=3, radial="spline")
    ref = osht.SHT(nside, lmax).map2alm(maps, niter=3)
    tri = np.array([ref[b, l, m] for b in range(nmaps) for l in range(lmax + 1) for m in range(l + 1)])
    e = rel_err(out.ravel(), tri)
    record(f"map2alm_{nmaps}maps_nside{nside}_lmax{lmax}_niter3", e)
    assert e < 1e-12


@pytest.mark.parametrize("nmaps", [1, 2, 3, 4, 12])
def test_map2alm_gram_refinement_vs_oracle(nmaps):
    """A geometry where most rings are alias-free (nside 32, lmax 40: the 20
    polar rings with nph <= 80 alias): the refinement passes run through the
    FP64 Gram matrices plus the aliased rings (matrix-vector kernels for 1, 2
    and 4 maps, tiled GEMMs for 3 and 12)."""
    nside, lmax = 32, 40
    a = sfbgpu.AnlmModes.from_nmax_lmax(1, lmax, 500.0, 1000.0, nside=nside, cache=True)
    rng = np.random.default_rng(10 + nmaps)
    maps = rng.normal(size=(nmaps, 12 * nside * nside)) + 2.0
    out = sfbgpu.cat2anlm.map2alm(maps, a, niter=3, radial="spline")
    ref = osht.SHT(nside, lmax).map2alm(maps, niter=3)
    tri = np.array([ref[b, l, m] for b in range(nmaps) for l in range(lmax + 1) for m in range(l + 1)])
    e = rel_err(out.ravel(), tri)
    record(f"map2alm_gram_{nmaps}maps_nside{nside}_lmax{lmax}_niter3", e)
    assert e < 1e-12


@pytest.mark.parametrize("zlim", [(0.5, 1.0), (-0.3, 0.3), (-1.0, -0.6)])
def test_map2alm_gram_partial_sky_vs_oracle(zlim):
    """Many maps that are zero outside a cap or band: the FP64 ring transform
    records the span of ring pairs with data and the first analysis pass sums
    over that span only."""
    nside, lmax, nmaps = 32, 40, 10
    a = sfbgpu.AnlmModes.from_nmax_lmax(1, lmax, 500.0, 1000.0, nside=nside, cache=True)
    rng = np.random.default_rng(40)
    th, _ = sfbgpu.pix2ang_ring(nside, np.arange(12 * nside * nside))
    z = np.cos(th)
    maps = (rng.normal(size=(nmaps, 12 * nside * nside)) + 2.0) * ((z > zlim[0]) & (z < zlim[1]))
    out = sfbgpu.cat2anlm.map2alm(maps, a, niter=3, radial="spline")
    ref = osht.SHT(nside, lmax).map2alm(maps, niter=3)
    tri = np.array([ref[b, l, m] for b in range(nmaps) for l in range(lmax + 1) for m in range(l + 1)])
    e = rel_err(out.ravel(), tri)
    record(f"map2alm_gram_partial_sky_z{zlim[0]}_{zlim[1]}", e)
    assert e < 1e-12


# ---------------------------------------------------------------- cat2amln ---
def _sep_window(a, nside, nr=50):
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, nside)
    phi = np.exp(-((wm.r - 750.0) / 200.0) ** 2)
    mask = sfbgpu.gen_mask(nside, 0.6)
    md = modes_dict(a, nside)
    m, wln = osfb.win_rhat_ln_separable(phi, mask, a.rmin, a.rmax, nr, md)
    return wm, phi, mask, wln


def test_cat2amln_spline_mode_vs_oracle(small):
    a = small
    md = modes_dict(a)
    rtp, w = catalogue(30_000, a.rmin, a.rmax, seed=3, weights=True, rpad=20.0)
    wm, phi, mask, wln = _sep_window(a, a.nside)
    nbar = rtp.shape[1] / (4 / 3 * np.pi * (a.rmax ** 3 - a.rmin ** 3))
    win = sfbgpu.SeparableArray(mask, wln, "mask", "w_ln")
    gpu = sfbgpu.cat2amln(rtp, a, nbar, win, w, radial="spline")
    ref = osfb.cat2amln(rtp, md, nbar, ("separable", mask, wln), w)
    record("cat2amln_spline_vs_reference_algorithm", rel_err(gpu, ref))
    assert rel_err(gpu, ref) < 1e-11


def test_cat2amln_poly_mode_vs_oracle(small):
    a = small
    md = modes_dict(a)
    rtp, w = catalogue(30_000, a.rmin, a.rmax, seed=4, weights=True, rpad=20.0)
    wm, phi, mask, wln = _sep_window(a, a.nside)
    nbar = rtp.shape[1] / (4 / 3 * np.pi * (a.rmax ** 3 - a.rmin ** 3))
    win = sfbgpu.SeparableArray(mask, wln, "mask", "w_ln")
    gpu = sfbgpu.cat2amln(rtp, a, nbar, win, w, radial="poly")
    ref = osfb.cat2amln(rtp, md, nbar, ("separable", mask, wln), w)
    info = sfbgpu.get_plan(a, radial="poly").info()
    e = rel_err(gpu, ref)
    record("cat2amln_poly_vs_reference_algorithm", e, radial_error=info["radial_error"],
           pieces=info["radial_pieces"], degree=info["radial_degree"])
    # interior spline interpolation error of the reference tables is ~4e-8 of max|g|
    assert info["radial_error"] < 1e-7
    assert e < 2e-7


@pytest.mark.parametrize("radial", ["spline", "poly"])
def test_cat2amln_dense_window_vs_oracle(small, radial):
    a = small
    md = modes_dict(a)
    nr = 40
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, a.nside)
    rng = np.random.default_rng(5)
    win = rng.random((nr, wm.npix))
    W = osfb.win_rhat_ln_dense(win, a.rmin, a.rmax, nr, md)
    rtp, _ = catalogue(10_000, a.rmin, a.rmax, seed=6)
    gpu = sfbgpu.cat2amln(rtp, a, 2e-4, W, None, radial=radial)
    ref = osfb.cat2amln(rtp, md, 2e-4, ("dense", W), None)
    record(f"cat2amln_dense_{radial}", rel_err(gpu, ref))
    assert rel_err(gpu, ref) < (1e-11 if radial == "spline" else 2e-7)


def test_cat2amln_empty_catalogue_zero_window(small):
    out = sfbgpu.cat2amln(np.zeros((3, 0)), small, 1.0, None)
    assert np.all(out == 0)


def test_cat2amln_errors(small):
    a = small
    rtp, _ = catalogue(100, a.rmin, a.rmax, seed=7)
    bad = rtp.copy()
    bad[0, 5] = np.nan
    with pytest.raises(capi.SFBError) as e:
        sfbgpu.cat2amln(bad, a, 1.0, None)
    assert e.value.status == capi.SFB_ENONFINITE
    bad = rtp.copy()
    bad[1, 3] = 4.0
    with pytest.raises(capi.SFBError) as e:
        sfbgpu.cat2amln(bad, a, 1.0, None)
    assert e.value.status == capi.SFB_ERANGE
    with pytest.raises(capi.SFBError) as e:
        sfbgpu.cat2amln(rtp, a, 0.0, None)
    assert e.value.status == capi.SFB_ENONFINITE
    # the plan stays usable after errors
    out = sfbgpu.cat2amln(rtp, a, 1.0, None)
    assert np.all(np.isfinite(out))


# ---------------------------------------------------------------- fields -----
def test_field2anlm_anlm2field_winrhat_vs_oracle(small):
    a = small
    md = modes_dict(a)
    nr = 60
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, a.nside)
    rng = np.random.default_rng(8)
    f = rng.normal(size=(nr, wm.npix))
    gpu = sfbgpu.field2anlm(f, wm, a)
    ref = osfb.field2anlm(f, a.rmin, a.rmax, nr, md)
    assert rel_err(gpu, ref) < 1e-11
    fb = sfbgpu.anlm2field(ref, wm, a)
    fr = osfb.anlm2field(ref, a.rmin, a.rmax, nr, md)
    assert rel_err(fb, fr) < 1e-11
    Wd = sfbgpu.win_rhat_ln(np.abs(f), wm, a)
    Wr = osfb.win_rhat_ln_dense(np.abs(f), a.rmin, a.rmax, nr, md)
    fin = np.isfinite(Wr)
    assert np.array_equal(fin, np.isfinite(Wd))
    assert rel_err(Wd[fin], Wr[fin]) < 1e-12
    phi = np.abs(f[:, 0])
    mask = np.ones(wm.npix)
    Ws = sfbgpu.win_rhat_ln(sfbgpu.SeparableArray(phi, mask, "phi", "mask"), wm, a)
    _, Wsr = osfb.win_rhat_ln_separable(phi, mask, a.rmin, a.rmax, nr, md)
    fin = np.isfinite(Wsr)
    assert rel_err(Ws.w_ln[fin], Wsr[fin]) < 1e-12


# ------------------------------------------- reference known-answer tests ----
def test_point_source_kat_nside256():
    """reference test/test_cat2anlm.jl:153-196 (nside 256, nmax 2, lmax 3, nr 100)."""
    a = sfbgpu.AnlmModes.from_nmax_lmax(2, 3, 500.0, 1000.0, nside=256)
    nr, ns = 100, 256
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, ns)
    f = np.zeros((nr, wm.npix))
    Op = 4 * np.pi / wm.npix
    for j in range(0, wm.npix, 3 * ns * ns + 7):
        for i in range(0, nr, 41):
            f[i, j] = 1
            an1 = round_sig(sfbgpu.field2anlm(f, wm, a), 6)
            th, ph = ohp.pix2ang_ring(ns, j)
            an0 = np.empty_like(an1)
            for k in range(1, sfbgpu.getnlmsize(a) + 1):
                n, l, m = sfbgpu.getnlm(a, k)
                g = a.basisfunctions(n, l, wm.r[i])
                an0[k - 1] = round_sig(wm.dr * wm.r[i] ** 2 * g * np.conj(ylm(l, m, th, ph)) * Op, 6)
            assert np.linalg.norm(an0 - an1) <= 1e-5 * max(np.linalg.norm(an0), np.linalg.norm(an1))
            f[i, j] = 0


@pytest.mark.parametrize("radial", ["spline", "poly"])
def test_basis_function_kat(radial):
    """reference test/test_cat2anlm.jl:32-67: window = g_nl Y^real_lm, -cat2amln(empty) = unit vector."""
    a = sfbgpu.AnlmModes(0.02, 0.0, 1000.0, nside=32)
    nr = 200
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, a.nside)
    th, ph = ohp.pix2ang_ring(32, np.arange(wm.npix))
    rng = np.random.default_rng(9)
    for idx in rng.integers(1, sfbgpu.getnlmsize(a) + 1, 6):
        n, l, m = sfbgpu.getnlm(a, int(idx))
        g = a.basisfunctions(n, l, wm.r)
        y = ylm(l, m, th, ph)
        yr = y.real if m == 0 else np.sqrt(2) * (-1) ** m * y.real
        W = sfbgpu.win_rhat_ln(np.outer(g, yr), wm, a, radial=radial)
        an = -sfbgpu.cat2amln(np.zeros((3, 0)), a, 3e-4, W, None, radial=radial)
        exp = 1 if m == 0 else (-1) ** m / np.sqrt(2)
        k = int(idx) - 1
        assert abs(an[k] - exp) < 1e-3
        assert np.max(np.abs(np.delete(an, k))) <= 2e-3


@pytest.mark.parametrize("radial", ["spline", "poly"])
def test_field2anlm_v1_equals_v2(radial):
    """reference test/test_cat2anlm.jl:235-258: -cat2amln(empty, win_rhat_ln(f)) == field2anlm(f)."""
    a = sfbgpu.AnlmModes.from_nmax_lmax(10, 10, 500.0, 1000.0, nside=32)
    wm = sfbgpu.ConfigurationSpaceModes.from_amodes(a, 100)
    f = np.random.default_rng(10).random((wm.nr, wm.npix))
    v1 = -sfbgpu.cat2amln(np.zeros((3, 0)), a, 1.0, sfbgpu.win_rhat_ln(f, wm, a), None, radial=radial)
    v2 = sfbgpu.field2anlm(f, wm, a)
    assert np.allclose(v1, v2, rtol=np.sqrt(np.finfo(float).eps), atol=0)


def test_anlm2field_round_trip():
    """reference test/test_cat2anlm.jl:261-289 (rtol 1e-4 after the first projection)."""
    a = sfbgpu.AnlmModes.from_nmax_lmax(10, 10, 500.0, 1000.0, nside=32)
    wm = sfbgpu.ConfigurationSpaceModes.from_amodes(a, 100)
    f1 = np.random.default_rng(11).random((wm.nr, wm.npix))
    a1 = sfbgpu.field2anlm(f1, wm, a)
    f2 = sfbgpu.anlm2field(a1, wm, a)
    a2 = sfbgpu.field2anlm(f2, wm, a)
    f3 = sfbgpu.anlm2field(a2, wm, a)
    a3 = sfbgpu.field2anlm(f3, wm, a)
    assert np.linalg.norm(f2 - f3) <= 1e-4 * np.linalg.norm(f2)
    assert np.linalg.norm(a1 - a2) <= 1e-4 * np.linalg.norm(a1)
    assert np.linalg.norm(a2 - a3) <= 1e-4 * np.linalg.norm(a2)


def test_amln2clnn_vs_oracle(small):
    """amln2clnn on the GPU (auto, cross, batched) vs the oracle restatement."""
    a = small
    md = modes_dict(a)
    cm = sfbgpu.ClnnModes(a, dnmax=2)
    rng = np.random.default_rng(12)
    x = rng.normal(size=(3, sfbgpu.getnlmsize(a))) + 1j * rng.normal(size=(3, sfbgpu.getnlmsize(a)))
    y = rng.normal(size=(3, sfbgpu.getnlmsize(a))) + 1j * rng.normal(size=(3, sfbgpu.getnlmsize(a)))
    auto = sfbgpu.amln2clnn(x[0], cm)
    cross = sfbgpu.amln2clnn(x, y, cm)
    assert rel_err(auto, osfb.amln2clnn(x[0], x[0], cm.lnn, md)) < 1e-14
    for b in range(3):
        assert rel_err(cross[b], osfb.amln2clnn(x[b], y[b], cm.lnn, md)) < 1e-14


def test_winweights2galweights_vs_oracle():
    """Bit-exact gather of per-galaxy weights from a shell x pixel field (src/cat2anlm.jl:218-238)."""
    nside, nr = 32, 40
    wm = sfbgpu.ConfigurationSpaceModes(500.0, 1000.0, nr, nside)
    rng = np.random.default_rng(13)
    W = rng.random((nr, wm.npix))
    rtp, _ = catalogue(100_000, 500.0, 1000.0, seed=14)
    rtp[0, :5] = [500.0, 1000.0, wm.r[3], sfbgpu.get_rbounds(wm)[7], 999.999999]
    gpu = sfbgpu.winweights2galweights(W, wm, rtp)
    ref = osfb.winweights2galweights(W, sfbgpu.get_rbounds(wm), nside, rtp)
    assert np.array_equal(gpu, ref)
    bad = rtp.copy()
    bad[0, 0] = 1001.0
    with pytest.raises(capi.SFBError) as e:
        sfbgpu.winweights2galweights(W, wm, bad)
    assert e.value.status == capi.SFB_ERANGE


@pytest.mark.parametrize("draws", ["uniform", "seed"])
def test_apply_window_vs_oracle(draws):
    """Device thinning (sfb_apply_window) against the oracle, bit-exact: the same
    kept galaxies in the same order, with the caller's draws or the library's
    counter-based stream; edge radii r == rmin, r == rmax and r beyond included."""
    nside, nr, rmin, rmax = 64, 40, 500.0, 1000.0
    wm = sfbgpu.ConfigurationSpaceModes(rmin, rmax, nr, nside)
    rng = np.random.default_rng(12)
    th, _ = sfbgpu.pix2ang_ring(nside, np.arange(wm.npix))
    win = np.exp(-((wm.r[:, None] - 750.0) / 150.0) ** 2) * (np.cos(th)[None, :] > -0.2)
    win = win * rng.uniform(0.5, 1.0, win.shape)
    rtp, _ = catalogue(300_000, rmin, rmax, seed=13, rpad=25.0)
    rtp[0, :4] = [rmin, rmax, rmin + 7 * wm.dr, rmax + 1e-9]
    n = rtp.shape[1]
    if draws == "uniform":
        u = rng.random(n)
        gpu = sfbgpu.apply_window(rtp, win, wm, uniform=u)
    else:
        u = osfb.splitmix64_uniform(2024, n)
        gpu = sfbgpu.apply_window(rtp, win, wm, seed=2024)
    ref = osfb.apply_window(rtp, win, rmin, rmax, wm.dr, nside, u)
    record(f"apply_window_{draws}_kept", float(gpu.shape[1]), of=n)
    assert gpu.shape == ref.shape and np.array_equal(gpu, ref)


# below one thread's 16 counters, one more, one tile of 4096 counters less one, many tiles: every odd size leaves the
# draws, which lie beside the counters, an odd number of doubles long
@pytest.mark.parametrize("n", [15, 17, 4095, 300_001])
def test_apply_window_odd_sizes(n):
    nside, nr, rmin, rmax = 16, 20, 500.0, 1000.0
    wm = sfbgpu.ConfigurationSpaceModes(rmin, rmax, nr, nside)
    rng = np.random.default_rng(n)
    win = rng.uniform(0.2, 1.0, (nr, wm.npix))
    rtp, _ = catalogue(n, rmin, rmax, seed=n)
    u = rng.random(n)
    gpu = sfbgpu.apply_window(rtp, win, wm, uniform=u)
    ref = osfb.apply_window(rtp, win, rmin, rmax, wm.dr, nside, u)
    assert gpu.shape == ref.shape and np.array_equal(gpu, ref)


def test_apply_window_edges():
    nside, nr = 4, 5
    wm = sfbgpu.ConfigurationSpaceModes(500.0, 1000.0, nr, nside)
    win = np.ones((nr, wm.npix))
    empty = sfbgpu.apply_window(np.zeros((3, 0)), win, wm)
    assert empty.shape == (3, 0)
    rtp = np.array([[700.0, 800.0], [1.0, 4.0], [0.5, 0.5]])        # theta > pi inside the shells
    with pytest.raises(capi.SFBError) as e:
        sfbgpu.apply_window(rtp, win, wm)
    assert e.value.status == capi.SFB_ERANGE
    bad = win.copy()
    bad[0, 0] = np.nan
    with pytest.raises(capi.SFBError) as e:
        sfbgpu.apply_window(rtp[:, :1], bad, wm)
    assert e.value.status == capi.SFB_ENONFINITE
    # every galaxy kept where win == max(win)
    rtp, _ = catalogue(1000, 500.0, 1000.0, seed=3)
    assert np.array_equal(sfbgpu.apply_window(rtp, win, wm, seed=1), rtp)


def test_win_lnn_vs_oracle():
    """W_l(n, n') of a window (radial selection x a mask tilted with
    direction) against the oracle's restatement of the reference: the shell
    a_00 from map2alm at 2 lmax, the trapezoidal radial sum.  FP64: 1e-12."""
    a = sfbgpu.AnlmModes(0.05, 500.0, 1000.0, nside=32)
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, 60, a.nside)
    th, ph = sfbgpu.pix2ang_ring(a.nside, np.arange(wm.npix))
    win = np.exp(-((wm.r[:, None] - 700.0) / 180.0) ** 2) * (1.0 + 0.3 * np.cos(th)[None, :]
                                                            + 0.1 * np.sin(3 * ph)[None, :] * np.sin(th)[None, :])
    cm = sfbgpu.ClnnModes(a, dnmax=3)
    gpu = sfbgpu.win_lnn(win, wm, cm)
    ref = osfb.win_lnn(win, a.rmin, a.rmax, wm.nr, modes_dict(a), cm.lnn)
    e = rel_err(gpu, ref)
    record("win_lnn_vs_oracle", e, nlnn=int(cm.lnn.shape[1]))
    assert e < 1e-12
    neg = win.copy()
    neg[3] = -1.0
    with pytest.raises(capi.SFBError) as ex:
        sfbgpu.win_lnn(neg, wm, cm)
    assert ex.value.status == capi.SFB_ENONFINITE


@pytest.mark.parametrize("neg_m", [False, True])
def test_calc_wmix_vs_oracle(neg_m):
    """The window mixing matrix against the oracle (exact Racah 3j symbols,
    FP64 map2alm of the window shells to 2 lmax): every entry, 1e-12 of the
    largest.  A constant full-sky window gives the radial overlap matrix:
    diagonal in (l, m), close to the identity in n."""
    a = sfbgpu.AnlmModes(0.02, 500.0, 1000.0, nside=8)
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, 40, a.nside)
    th, ph = sfbgpu.pix2ang_ring(a.nside, np.arange(wm.npix))
    win = np.exp(-((wm.r[:, None] - 700.0) / 180.0) ** 2) * (1.0 + 0.3 * np.cos(th)[None, :]
                                                            + 0.2 * np.sin(2 * ph)[None, :] * np.sin(th)[None, :] ** 2)
    gpu = sfbgpu.calc_wmix(win, wm, a, neg_m=neg_m)
    ref = osfb.calc_wmix(win, a.rmin, a.rmax, wm.nr, modes_dict(a), neg_m=neg_m)
    e = rel_err(gpu, ref)
    record(f"calc_wmix_vs_oracle_negm{int(neg_m)}", e, nlmsize=int(gpu.shape[0]))
    assert np.all(np.isfinite(gpu)) and e < 1e-12
    if not neg_m:
        # A constant window: nside 16 so that the window's band limit 2 lmax = 30 stays below
        # 2 nside (at nside 8 the ring quadrature of L > 2 nside leaves a 3% diagonal error,
        # in the oracle too); 400 shells put the midpoint rule of the overlaps near 1e-5.
        a16 = sfbgpu.AnlmModes(0.02, 500.0, 1000.0, nside=16)
        wf = sfbgpu.ConfigurationSpaceModes(a16.rmin, a16.rmax, 400, a16.nside)
        one = sfbgpu.calc_wmix(np.ones((wf.nr, wf.npix)), wf, a16)
        dev = float(np.max(np.abs(one - np.eye(one.shape[0]))))
        record("calc_wmix_constant_window_identity", dev, nside=16, shells=400)
        assert dev < 1e-4
