"""Cells so large that squared distances leave the FP32 range: the cutoff pre-test of the
real-space kernels must hand every pair to the exact test then.

The sums scale with the cell (velocities of forces do not change, those of the stresslet
fall with its side), so a cell of 2^66 is held against one of 1.  All values scale by
powers of two, and the all-FP64 form must agree to rounding: 1e-13.  The default form's
float-float pairs have FP32's range themselves; with one box (side 1, every pair
near) they play no part, and it must agree as well."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
SCALE = 2.0 ** 66


@pytest.fixture(scope="module")
def ft():
    import fasttools2d_gb300 as ft
    return ft


def _cloud(N, nt):
    rng = np.random.default_rng(3)
    p, q = rng.random((2, N)) - 0.5, rng.random((2, nt)) - 0.5
    th = rng.random(N) * 2 * np.pi
    return p, q, rng.standard_normal((2, N)), np.vstack([np.cos(th), np.sin(th)])


@pytest.mark.parametrize("precision,nside", [("fp64_native", 1), ("fp64_native", 3), ("fp64_native", 7), ("fp64", 1)])
def test_real_space(ft, precision, nside):
    p, q, f, n = _cloud(3000, 2000)
    xi = 5 * nside / 3
    plan = ft.Plan(0)
    plan.set_precision(precision)
    for fn, args, s in ((ft.mex_stokes_slp_real, (f,), 1.0), (ft.mex_stokes_dlp_real, (f, n), SCALE)):
        want = fn(p, q, *args, xi, nside, nside, 1.0, 1.0, plan=plan)
        got = fn(p * SCALE, q * SCALE, *args, xi / SCALE, nside, nside, SCALE, SCALE, plan=plan)
        assert relerr(got * s, want) < 1e-13, (fn.__name__, relerr(got * s, want))
    plan.close()


@pytest.mark.parametrize("nside", [1, 3, 7])
def test_gradients(ft, nside):
    p, q, f, _ = _cloud(1000, 800)
    w = np.random.default_rng(4).standard_normal((2, 800))
    plan = ft.Plan(0)
    plan.set_precision("fp64_native")
    grads = []
    for s in (1.0, SCALE):
        prm = ft.EwaldParams.derived(5 * nside / 3 / s, nside, nside, 64, 64, 24, s, s)
        gp, gf, _, _ = ft.stokes_ewald_adjoint(p * s, q * s, f, None, None, w, None, prm, plan=plan)
        grads += [gp * s, gf]
    assert relerr(grads[2], grads[0]) < 1e-12 and relerr(grads[3], grads[1]) < 1e-12
    plan.close()
