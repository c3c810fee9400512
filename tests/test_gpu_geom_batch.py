"""A batch of densities of which some take the FP64 spread: the tile lists of the
tensor-core spread are built once for all of them, whichever density is the one that
does not use them.

Tolerances: 3e-13 against single evaluations (as in test_gpu_geom.py), and 1e-11 where
both sides ran the FP64 spread, whose atomics add in varying order."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
SINGLE, ATOMICS = 3e-13, 1e-11


@pytest.fixture(scope="module")
def ft():
    import fasttools2d_gb300 as ft
    return ft


def _cloud(N, seed, nrhs):
    rng = np.random.default_rng(seed)
    p, q = rng.random((2, N)), rng.random((2, N))
    th = rng.random(N) * 2 * np.pi
    return p, q, np.vstack([np.cos(th), np.sin(th)]), rng.standard_normal((nrhs, 2, N))


@pytest.mark.parametrize("bad", [(0,), (0, 1), (2,), (0, 1, 2, 3)])
@pytest.mark.parametrize("what", ["nan", "inf"])
def test_non_finite_densities(ft, bad, what):
    N = 6000
    p, q, n, f = _cloud(N, 5 + len(bad), 4)
    for r in bad:
        f[r, 0, 123 + r] = np.nan if what == "nan" else np.inf
    prm = ft.EwaldParams.derived(60.0, 12, 12, 96, 96, 24, 1.0, 1.0)
    plan, one = ft.Plan(0), ft.Plan(0)          # (a plan without lists of earlier calls)
    geo = ft.Geometry(p, q, prm, n=n, plan=plan)
    us, ud = geo.apply(f, f)
    for r in range(4):
        vs, vd = ft.stokes_ewald(p, q, f[r], f[r], n, prm, plan=one)
        assert np.array_equal(np.isfinite(us[r]), np.isfinite(vs))
        if r not in bad:
            assert np.isfinite(us[r]).all() and np.isfinite(ud[r]).all()
            assert relerr(us[r], vs) < SINGLE and relerr(ud[r], vd) < SINGLE
    geo.close()
    plan.close()
    one.close()


@pytest.mark.parametrize("dense", [(0,), (1,), (0, 2)])
def test_crowded_and_sparse_densities(ft, dense):
    """30,000 sources in one grid cell: a density on all of them takes the FP64 spread
    (more than 2^14 cover a node), one on 1000 of them the integer one."""
    N = 30000
    p, q, n, f = _cloud(N, 11, 3)
    p = -0.3 + p / 128
    for r in range(3):
        if r not in dense:
            f[r, :, 1000:] = 0.0
    prm = ft.EwaldParams.derived(40.0, 8, 8, 128, 128, 24, 1.0, 1.0)
    plan, one = ft.Plan(0), ft.Plan(0)
    geo = ft.Geometry(p, q, prm, kinds="slp", plan=plan)
    us, _ = geo.apply(f)
    for r in range(3):
        vs = ft.slp_ewald(p, q, f[r], prm, plan=one)
        assert relerr(us[r], vs) < (ATOMICS if r in dense else SINGLE), (r, relerr(us[r], vs))
    geo.close()
    plan.close()
    one.close()
