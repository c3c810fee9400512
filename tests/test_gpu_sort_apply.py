"""The fused wrap, box and sort kernels where their fast paths end (box edges,
points periods away, more boxes than one scan's blocks take), and the geometry's
operator product at each number of warps per slice of rows."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
PARITY = 1e-12


@pytest.fixture(scope="module")
def ft():
    import fasttools2d_gb300 as ft
    return ft


@pytest.mark.parametrize("L,nx,ny", [((1.0, 1.0), 7, 7), ((0.7, 1.4), 5, 10), ((3.0, 3.0), 8, 8)])
def test_wrap_and_boxes_on_their_edges(ft, L, nx, ny):
    """Coordinates on and beside box edges and half periods, up to 5 periods out,
    against the oracle's wrap and box assignment."""
    from oracle import oracle as O
    rng = np.random.default_rng(nx)
    def coords(Lc, n):
        e = np.array([k * Lc / n - Lc / 2 for k in range(n + 1)] + [0.0, Lc / 2, Lc, 1.5 * Lc, -Lc])
        e = np.concatenate([e, np.nextafter(e, 9), np.nextafter(e, -9), e + 3 * Lc, e - 5 * Lc,
                            [-1e-20, 1e-20, -1e-300]])
        return rng.permutation(np.concatenate([e, Lc * (rng.random(200) * 9 - 4)]))[:200]
    p = np.vstack([coords(L[0], nx)[:150], coords(L[1], ny)[:150]])
    q = np.vstack([coords(L[0], nx)[:140], coords(L[1], ny)[:140]])
    f = rng.standard_normal((2, 150))
    xi = 4.8 * nx / L[0]
    M = 64
    prm = ft.EwaldParams.derived(xi, nx, ny, M, M * round(L[1] / L[0]), 24, *L)
    plan = ft.Plan(0)
    u = ft.slp_ewald(p, q, f, prm, plan=plan)
    plan.close()
    v = O.slp_ewald(p, q, f, xi, nx, ny, M, M * round(L[1] / L[0]), *L, 24)[0]
    assert np.array_equal(np.isnan(u), np.isnan(v))
    assert relerr(np.nan_to_num(u), np.nan_to_num(v)) < PARITY


@pytest.mark.parametrize("nside", [32, 33, 362, 363, 500])
def test_sort_into_many_boxes(ft, nside):
    """Numbers of boxes around 1024 and 2^17 (one block scans them all beyond)."""
    from oracle import oracle as O
    rng = np.random.default_rng(nside)
    p, q = rng.random((2, 3000)) - 0.5, rng.random((2, 2000)) - 0.5
    q[:, :1000] = p[:, :1000] + 0.3 / nside
    q = np.clip(q, -0.5, 0.4999)
    f = rng.standard_normal((2, 3000))
    plan = ft.Plan(0)
    u = ft.mex_stokes_slp_real(p, q, f, 4.8 * nside, nside, nside, 1.0, 1.0, plan=plan)
    plan.close()
    assert relerr(u, O.mex_stokes_slp_real(p, q, f, 4.8 * nside, nside, nside, 1.0, 1.0)) < PARITY


@pytest.mark.parametrize("nt", [33, 40000, 80000, 156000])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_geometry_apply_warps_per_slice(ft, nt, nrhs):
    """8, 4, 2 and 1 warps per slice of 32 rows."""
    rng = np.random.default_rng(nt)
    ns = 2000
    p, q = rng.random((2, ns)), rng.random((2, nt))
    th = rng.random(ns) * 2 * np.pi
    n = np.vstack([np.cos(th), np.sin(th)])
    f, g = rng.standard_normal((2, nrhs, 2, ns))
    prm = ft.EwaldParams.derived(28.8, 6, 6, 96, 96, 24, 1.0, 1.0)
    plan = ft.Plan(0)
    us, ud = ft.Geometry(p, q, prm, n=n, plan=plan).apply(f, g)
    for r in range(nrhs):
        vs, vd = ft.stokes_ewald(p, q, f[r], g[r], n, prm, plan=plan)
        assert relerr(us[r], vs) < 3e-13 and relerr(ud[r], vd) < 3e-13
    plan.close()
