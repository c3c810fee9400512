"""Cells in small units.  The reference takes a point within 1e-13 of a grid node as lying
on it, whatever the node spacing (ewald_tools.cpp:86-114), so that in cells of 1e-5 or 1e-9
a visible share of points is moved; the default form's stencils must be moved like
those of the all-FP64 form.  Tolerance: 1e-13, gradients 1e-11, as in the other k-space
tests."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plans():
    import fasttools2d_gb300 as ft
    a, nat = ft.Plan(0), ft.Plan(0)
    nat.set_precision("fp64_native")
    yield a, nat
    a.close()
    nat.close()


@pytest.mark.parametrize("L,M", [(1.0, 128), (1e-5, 256), (1e-7, 128), (2.0 ** -30, 128), (1e-11, 128)])
def test_snapped_points(plans, L, M):
    import fasttools2d_gb300 as ft
    P = 24
    rng = np.random.default_rng(5)
    h = L / M

    def points(n):
        # on nodes and within three snapping distances of them, and anywhere
        i = rng.integers(-M // 2, M // 2, (2, n)) * h
        d = np.clip(rng.uniform(-3e-13, 3e-13, (2, n)), -0.4 * h, 0.4 * h)
        p = np.where(rng.random((2, n)) < 0.1, i, i + d)
        return np.where(rng.random((2, n)) < 0.3, (rng.random((2, n)) - 0.5) * L, p)

    p, q = points(3000), points(2000)
    th = rng.random(3000) * 2 * np.pi
    n, f = np.vstack([np.cos(th), np.sin(th)]), rng.standard_normal((2, 3000))
    w = P * h / 2
    xi = 0.9 * np.sqrt(np.pi * P) / (2 * w)
    for fn, args in ((ft.mex_stokes_slp_kspace, (f,)), (ft.mex_stokes_dlp_kspace, (f, n))):
        a, b = (fn(p, q, xi, 0.9, *args, M, M, L, L, w, P, plan=pl) for pl in plans)
        assert relerr(a, b) < 1e-13, (fn.__name__, relerr(a, b))
    prm = ft.EwaldParams(xi, 8, 8, M, M, P, L, L, w, 0.9)
    g = [ft.stokes_ewald_adjoint(p, q, f, None, None, rng.standard_normal((2, 2000)) * 0 + 1, None, prm, plan=pl)
         for pl in plans]
    assert relerr(g[0][1], g[1][1]) < 1e-11, relerr(g[0][1], g[1][1])
