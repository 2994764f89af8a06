"""The FP64 contractions on the tensor cores (many columns, Legendre and ring
transforms) at the edges of their tiles, against the oracle's map2alm and against the plan's FP64 units
(SFBGPU_TC64=0, SFBGPU_RING64=0).

Tolerance: a value is held to half a unit of 2^-55 of its column's (table
row's) largest magnitude, and the level sums lose less than that again, so a
sum over K values is off by at most about K 2^-54 max|F| max|lambda|.  For
N(0, 1) maps max|F| is about 4 rms and a coefficient is about sqrt(K) times
the product of the rms values: sqrt(1024) * 16 * 2^-54 = 3e-14 of max|a| a
pass, 1e-13 over the four passes of niter = 3."""

import numpy as np
import pytest

import sfbgpu
from helpers import record, rel_err
from oracle.sht import SHT
from sfbgpu.cat2anlm import map2alm, map2alm_adjoint

pytestmark = pytest.mark.gpu
TOL = 1e-13


def _modes(lmax, nside):
    return sfbgpu.AnlmModes.from_nmax_lmax(1, lmax, 500.0, 1000.0, nside=nside, cache=True)


def _maps(nmaps, nside, seed):
    return np.random.default_rng(seed).normal(size=(nmaps, 12 * nside * nside))


# lmax: 16-row padding (30: 16 rows, 31, 32: 17), the 64-row tile (126: 64 rows, 128: 65); nmaps: a
# partial 128-column tile, a whole one, one column more; nside 8: one 16-ring chunk, 12: a ragged one
@pytest.mark.parametrize("nside,lmax,nmaps,niter", [(8, 16, 5, 0), (8, 15, 7, 3), (12, 30, 5, 3), (16, 31, 64, 3),
                                                    (16, 32, 65, 0), (32, 63, 9, 3), (64, 126, 6, 0),
                                                    (64, 128, 6, 3)])
def test_edges_vs_oracle(nside, lmax, nmaps, niter):
    a = _modes(lmax, nside)
    f = _maps(nmaps, nside, lmax)
    ref = SHT(nside, lmax).map2alm(f, niter=niter)
    ref = np.stack([ref[:, l, m] for l in range(lmax + 1) for m in range(l + 1)], axis=1)
    e = rel_err(map2alm(f, a, niter=niter, radial="spline"), ref)
    record(f"fp64_tc_map2alm_{nside}_{lmax}_{nmaps}_{niter}", e)
    assert e < TOL


# more than 256 ring pairs (the sum runs in exact blocks of 256), more than 64 and 128 rows
@pytest.mark.parametrize("nside,lmax,nmaps", [(128, 256, 5), (160, 140, 5), (256, 300, 6)])
def test_long_sums_vs_fp64_units(nside, lmax, nmaps, monkeypatch):
    f = _maps(nmaps, nside, 3)
    got = map2alm(f, _modes(lmax, nside), radial="spline")
    monkeypatch.setenv("SFBGPU_TC64", "0")
    ref = map2alm(f, _modes(lmax, nside), radial="spline")
    e = rel_err(got, ref)
    record(f"fp64_tc_long_{nside}_{lmax}", e)
    assert e < TOL


@pytest.mark.parametrize("nside,lmax,nmaps,niter", [(16, 24, 9, 3), (16, 40, 65, 0), (32, 60, 33, 3), (16, 60, 6, 2)])
def test_adjoint_vs_fp64_units(nside, lmax, nmaps, niter, monkeypatch):
    """(16, 60): most rings alias, so the refinement runs over every ring."""
    rng = np.random.default_rng(7)
    n = (lmax + 1) * (lmax + 2) // 2
    y = rng.normal(size=(nmaps, n)) + 1j * rng.normal(size=(nmaps, n))
    got = map2alm_adjoint(y, _modes(lmax, nside), niter=niter, radial="spline")
    monkeypatch.setenv("SFBGPU_TC64", "0")
    ref = map2alm_adjoint(y, _modes(lmax, nside), niter=niter, radial="spline")
    e = rel_err(got, ref)
    record(f"fp64_tc_adjoint_{nside}_{lmax}_{nmaps}", e)
    assert e < TOL


@pytest.mark.parametrize("nmaps", [1, 2, 3, 4])
@pytest.mark.parametrize("nside,lmax", [(16, 24), (32, 60), (12, 30)])
def test_few_maps(nside, lmax, nmaps):
    """Up to eight columns take their own kernels (the oracle, as above), whatever the plan has done before: the
    same bits before and after a call of many columns."""
    a = _modes(lmax, nside)
    f = _maps(nmaps, nside, 8)
    first = map2alm(f, a, radial="spline")
    ref = SHT(nside, lmax).map2alm(f, niter=3)
    ref = np.stack([ref[:, l, m] for l in range(lmax + 1) for m in range(l + 1)], axis=1)
    assert rel_err(first, ref) < TOL
    y = np.random.default_rng(9).normal(size=(nmaps, ref.shape[1], 2)) @ np.array([1.0, 1j])
    back = map2alm_adjoint(y, a, radial="spline")
    map2alm(_maps(9, nside, 8), a, radial="spline")
    assert np.array_equal(map2alm(f, a, radial="spline"), first)
    assert np.array_equal(map2alm_adjoint(y, a, radial="spline"), back)


@pytest.mark.parametrize("scale", [1e-25, 1e30])
def test_scales(scale):
    """Magnitudes far from one (the ring transform's odd factors run in double-float, which bounds them)."""
    a = _modes(24, 16)
    f = _maps(6, 16, 5)
    one = map2alm(f, a, radial="spline")
    e = rel_err(map2alm(f * scale, a, radial="spline") / scale, one)
    assert e < 1e-13


def _per_m(a, lmax):
    """The largest magnitude of each m: [map, l (l+1)/2 + m] -> [map, m]."""
    m = np.concatenate([np.arange(l + 1) for l in range(lmax + 1)])
    return np.stack([np.max(np.abs(a[:, m == k]), axis=1) for k in range(lmax + 1)], axis=1)


# the sum over the rings in one launch of many chunks, with 2 and with 16, and (16, 24) in resident chunks
@pytest.mark.parametrize("nside,lmax", [(16, 24), (64, 120), (256, 90)])
@pytest.mark.parametrize("units", ["SFBGPU_TC64", "SFBGPU_RING64"])
def test_bright_pixels_near_a_pole(nside, lmax, units, monkeypatch):
    """Two pixels of 1e8 on the shortest rings, whose spectra reach every m, on N(0, 1) noise: each m on its own scale
    is as close to the FP64 units as maps without them (the tolerance above).  The refinement passes through sums
    over m, which the 1e8 at m = 0 leaves uncertain at 5e-11 of the others (the same in FP64 against 80 bits): 1e-10."""
    f = _maps(6, nside, 21)
    f[:, 1] += 1e8
    f[:, 17] -= 1e8
    for niter, tol in ((0, TOL), (3, 1e-10)):
        monkeypatch.delenv(units, raising=False)
        got = map2alm(f, _modes(lmax, nside), niter=niter, radial="spline")
        monkeypatch.setenv(units, "0")
        ref = map2alm(f, _modes(lmax, nside), niter=niter, radial="spline")
        e = float(np.max(_per_m(got - ref, lmax) / _per_m(ref, lmax)))
        record(f"fp64_bright_{units}_{nside}_{lmax}_{niter}", e)
        assert e < tol, (niter, e)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite_and_zero_maps(bad, monkeypatch):
    """A non-finite map spoils its own coefficients, as on the FP64 units, and no other map's."""
    f = _maps(9, 16, 6)
    f[3, 100] = bad
    f[5] = 0.0
    got = map2alm(f, _modes(24, 16), radial="spline")
    monkeypatch.setenv("SFBGPU_TC64", "0")
    ref = map2alm(f, _modes(24, 16), radial="spline")
    assert np.array_equal(np.isfinite(got), np.isfinite(ref)) and not np.isfinite(got[3]).any()
    ok = [i for i in range(9) if i != 3]
    assert rel_err(got[ok], ref[ok]) < TOL
    assert not np.any(got[5])


# rings from 4 pixels on (nside 2), an nside that is no power of two, n/4 at and next to multiples of the
# 16-value chunk and the 32-value tile, more than 192 values (two exact blocks), 2 lmax above and below the
# ring lengths, a partial and a whole tile of 64 maps and one map more
@pytest.mark.parametrize("nside,lmax,nmaps", [(2, 3, 5), (2, 8, 5), (3, 4, 6), (5, 14, 9), (15, 30, 64), (16, 31, 65),
                                              (17, 33, 7), (31, 64, 5), (32, 20, 33), (33, 62, 5), (64, 63, 5),
                                              (192, 60, 5), (256, 127, 5)])
def test_rings_vs_fft(nside, lmax, nmaps, monkeypatch):
    f = _maps(nmaps, nside, 11)
    f[1] = 0.0
    f[2, : 6 * nside * nside] = 0.0                   # rings without data in some maps
    f[3, 5 * nside * nside] += 1e6                    # a spike
    y = np.random.default_rng(12).normal(size=(nmaps, (lmax + 1) * (lmax + 2) // 2, 2)) @ np.array([1.0, 1j])
    y[1] = 0.0
    a = _modes(lmax, nside)
    got = map2alm(f, a, niter=0, radial="spline"), map2alm_adjoint(y, a, niter=0, radial="spline")
    monkeypatch.setenv("SFBGPU_RING64", "0")
    b = _modes(lmax, nside)
    ref = map2alm(f, b, niter=0, radial="spline"), map2alm_adjoint(y, b, niter=0, radial="spline")
    for g, r, what in zip(got, ref, ("analysis", "synthesis")):
        for k in range(nmaps):                        # each map on its own scale
            e = float(np.max(np.abs(g[k] - r[k])) / max(np.max(np.abs(r[k])), 1e-300))
            record(f"fp64_ring_{what}_{nside}_{lmax}_map{k}", e)
            assert e < TOL, (what, k, e)


def test_pixel_major_fields_vs_fft(monkeypatch):
    """anlm2field and the field gradient (FP64 and FP32) write their fields straight from the ring transform."""
    rng = np.random.default_rng(13)
    out = []
    for v in ("1", "0"):
        monkeypatch.setenv("SFBGPU_RING64", v)
        a = sfbgpu.AnlmModes(0.03, 500.0, 1000.0, nside=16)
        wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, 37, 16)
        n = sfbgpu.getnlmsize(a)
        c = np.random.default_rng(14).normal(size=(n, 2)) @ np.array([1.0, 1j])
        out.append([sfbgpu.anlm2field(c, wm, a)] + [sfbgpu.cat2anlm.field2anlm_vjp(c, wm, a, dtype=d)
                                                    for d in (np.float64, np.float32)])
    for g, r in zip(*out):
        assert g.shape == r.shape and g.dtype == r.dtype
        assert rel_err(g, r) < (TOL if g.dtype == np.float64 else 1e-6)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_rings_nonfinite(bad, monkeypatch):
    f = _maps(6, 16, 15)
    f[2, 40] = bad
    y = np.ones((6, 25 * 26 // 2), complex)
    y[4, 7] = bad
    a = _modes(24, 16)
    g = map2alm(f, a, radial="spline"), map2alm_adjoint(y, a, radial="spline")
    assert not np.isfinite(g[0][2]).any() and np.isfinite(np.delete(g[0], 2, 0)).all()
    assert not np.isfinite(g[1][4]).any() and np.isfinite(np.delete(g[1], 4, 0)).all()


# 50 MB in three belt groups and the caps; the caps and the belt share a table tile, or (nside 65) just do not
@pytest.mark.parametrize("nside,nr", [(64, 129), (65, 129)])
def test_large_synthesis_in_ring_groups(nside, nr, monkeypatch):
    """anlm2field with the Legendre synthesis ring group by ring group against the FP64 units in one launch."""
    out = []
    for v in ("1", "0"):
        monkeypatch.setenv("SFBGPU_TC64", v)
        a = sfbgpu.AnlmModes(0.054, 500.0, 1500.0, nside=nside)
        assert 2 * (a.lmax + 1) * ((2 * nr + 127) // 128) >= 304
        wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, nside)
        c = np.random.default_rng(16).normal(size=(sfbgpu.getnlmsize(a), 2)) @ np.array([1.0, 1j])
        out.append(sfbgpu.anlm2field(c, wm, a))
    assert rel_err(out[0], out[1]) < TOL


# shells below, at and above the four warps' terms and the chunks of 16 they stage, in one chunk and in several
@pytest.mark.parametrize("nr", [1, 2, 3, 5, 63, 64, 65, 70])
def test_few_shells_vs_map2alm(nr):
    """The radial sum over few shells: sum_s r_s^2 dr g_nl(r_s) a_lm(s) of the shells' own transforms, FP64.
    A different grouping of at most 70 FP64 terms: 1e-12."""
    a = sfbgpu.AnlmModes(0.03, 500.0, 1000.0, nside=16)
    wm = sfbgpu.ConfigurationSpaceModes(a.rmin, a.rmax, nr, 16)
    f = np.asfortranarray(np.random.default_rng(17).normal(size=(nr, wm.npix)))
    whole = sfbgpu.field2anlm(f, wm, a, precision="fp64")
    parts = np.zeros_like(whole)
    for s in range(nr):                                # linear in the shells
        one = np.zeros_like(f)
        one[s] = f[s]
        parts += sfbgpu.field2anlm(one, wm, a, precision="fp64")
    assert rel_err(whole, parts) < 1e-12
