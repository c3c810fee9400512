"""k-space sums on grids whose lengths take each kind of row transform.

Lengths that take each radix, alone and after others, and some with a prime above 7 in
one or both directions, against the oracle.  The bound is
the parity bound of the other k-space comparisons (1e-12): a row transform in
float-float errs by a few 2^-46 of the row's largest value."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
PARITY = 1e-12


@pytest.mark.parametrize("Mx,My", [(144, 60), (36, 84), (420, 48), (640, 96), (72, 350), (486, 98),
                                   (132, 72), (276, 92), (104, 64)])
def test_kspace_on_grid_lengths(Mx, My):
    import fasttools2d_gb300 as ft
    from oracle import oracle as O
    rng = np.random.default_rng(Mx * 1000 + My)
    Lx, P = 1.0, 20
    Ly = My / Mx
    ps = np.vstack([rng.random(150) * Lx, rng.random(150) * Ly])
    pt = np.vstack([rng.random(90) * Lx, rng.random(90) * Ly])
    f, g, n = (rng.standard_normal((2, 150)) for _ in range(3))
    w = P * Lx / Mx / 2
    xi = 0.25 * Mx
    eta = (2 * xi * w / (0.95 * np.sqrt(np.pi * P))) ** 2
    plan = ft.Plan(0)
    try:
        got = ft.mex_stokes_slp_kspace(ps, pt, xi, eta, f, Mx, My, Lx, Ly, w, P, plan=plan)
        assert relerr(got, O.mex_stokes_slp_kspace(ps, pt, xi, eta, f, Mx, My, Lx, Ly, w, P)) < PARITY
        got = ft.mex_stokes_dlp_kspace(ps, pt, xi, eta, f, n, Mx, My, Lx, Ly, w, P, plan=plan)
        assert relerr(got, O.mex_stokes_dlp_kspace(ps, pt, xi, eta, f, n, Mx, My, Lx, Ly, w, P)) < PARITY
    finally:
        plan.close()
