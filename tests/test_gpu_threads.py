"""Plans of different sizes on several threads, one plan each."""

import threading

import numpy as np
import pytest

import sfbgpu
from sfbgpu.cat2anlm import map2alm_adjoint

pytestmark = pytest.mark.gpu


def test_kernels_shared_by_plans_of_different_sizes():
    """The same kernels with 70 to 215 KB of shared memory, launched by four threads at once: every call succeeds and
    gives the bits that it gives alone."""
    work = []
    for nside, lmax in ((16, 40), (20, 70), (32, 120), (43, 170)):
        a = sfbgpu.AnlmModes.from_nmax_lmax(1, lmax, 500.0, 1000.0, nside=nside, cache=True)
        rng = np.random.default_rng(lmax)
        y = rng.normal(size=(5, (lmax + 1) * (lmax + 2) // 2, 2)) @ np.array([1.0, 1j])
        work.append((a, y, map2alm_adjoint(y, a, niter=0, radial="spline")))
    wrong = []

    def go(a, y, alone):
        try:
            for _ in range(1500):
                if not np.array_equal(map2alm_adjoint(y, a, niter=0, radial="spline"), alone):
                    wrong.append((a.lmax, "differs"))
                    return
        except Exception as e:
            wrong.append((a.lmax, str(e)))

    threads = [threading.Thread(target=go, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
