"""Calls at the limits of the device memory: what fits one after another still runs when it does not fit together."""

import gc

import numpy as np
import pytest

import sfbgpu
from helpers import rel_err
from sfbgpu.cat2anlm import map2alm, map2alm_adjoint
from test_gpu_batched import _mocks, _window

pytestmark = pytest.mark.gpu


def _free():
    import torch
    gc.collect()                                       # plans of earlier tests
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _leave(nbytes):
    """Device memory held so that about nbytes are left."""
    import torch
    return torch.empty(max(_free() - int(nbytes), 1), dtype=torch.uint8, device="cuda")


def _roomy_and_tight(call, step):
    """call(amodes) on a plan with all the memory there is, and on new ones with less and less left, by steps of that
    part of what the first took, until one holds less: the first and the last result."""
    def run(left):
        a = sfbgpu.AnlmModes(0.03, 500.0, 1000.0, nside=64)
        plan = sfbgpu.get_plan(a, precision="mixed")
        tables = plan.info()["device_bytes"]
        held = None if left is None else _leave(left)
        try:
            return call(a), plan.info()["device_bytes"] - tables
        finally:
            del held
            plan.close()
            _free()

    run(None)                                          # (kernels are loaded at their first launch)
    roomy, most = run(None)
    for k in range(20):
        tight, used = run((1.05 - k * step) * most)
        if used < most:
            return roomy, tight
    raise AssertionError("there was always room")


def test_dense_window_beside_the_basis_maps():
    """The joint transform of basis and window maps does not fit: first the ones, then the others (mixed: 1e-9)."""
    a = sfbgpu.AnlmModes(0.03, 500.0, 1000.0, nside=64)
    wm, phi, mask = _window(a)
    sep = sfbgpu.SeparableArray(phi, mask, "phi", "mask")
    win = sfbgpu.win_rhat_ln(sep.dense(), wm, a)
    (rtp,), (w,) = _mocks(a, [5000], 61)
    nbar = 5000 / sfbgpu.integrate_window(sep, wm)

    one, two = _roomy_and_tight(lambda m: sfbgpu.cat2amln(rtp, m, nbar, win, w, precision="mixed"), 0.015)
    assert rel_err(two, one) < 1e-9


def test_group_of_mocks():
    """The workspace of a group does not fit: its mocks one by one."""
    a = sfbgpu.AnlmModes(0.03, 500.0, 1000.0, nside=64)
    wm, phi, mask = _window(a)
    sep = sfbgpu.SeparableArray(phi, mask, "phi", "mask")
    win = sfbgpu.win_rhat_ln(sep, wm, a)
    sizes = [3000, 0, 2500, 4100, 1, 3300, 2800, 1999, 3000, 3000]
    cats, ws = _mocks(a, sizes, 67)
    nbars = [max(n, 1) / sfbgpu.integrate_window(sep, wm) for n in sizes]

    one, two = _roomy_and_tight(lambda m: sfbgpu.cat2amln_batched(cats, m, nbars, win, ws, precision="mixed"), 0.05)
    for x, y in zip(one, two):
        assert rel_err(y, x) < 1e-9 or not np.any(x)


def test_tables_are_made_when_there_is_memory():
    """A plan whose first calls find no memory for the digit tables runs them on the FP64 units (1e-13, as the
    tensor-core tests) and later ones as any other plan: the same bits."""
    def modes():
        return sfbgpu.AnlmModes.from_nmax_lmax(1, 60, 500.0, 1000.0, nside=64, cache=True)

    f = np.random.default_rng(5).normal(size=(6, 12 * 64 * 64))
    y = np.random.default_rng(6).normal(size=(6, 61 * 62 // 2, 2)) @ np.array([1.0, 1j])
    a, b = modes(), modes()
    fresh = map2alm(f, b, radial="spline"), map2alm_adjoint(y, b, radial="spline")
    before = sfbgpu.get_plan(a, radial="spline").info()["device_bytes"]
    held = _leave(60e6)                                # the tables take more than a sixteenth of this
    short = map2alm(f, a, radial="spline"), map2alm_adjoint(y, a, radial="spline")
    small = sfbgpu.get_plan(a, radial="spline").info()["device_bytes"]
    del held
    _free()
    later = map2alm(f, a, radial="spline"), map2alm_adjoint(y, a, radial="spline")
    assert sfbgpu.get_plan(a, radial="spline").info()["device_bytes"] > small > before
    for s, l, g in zip(short, later, fresh):
        assert rel_err(s, g) < 1e-13 and np.array_equal(l, g)
