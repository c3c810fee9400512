"""The tensor-core spread and gather against the all-FP64 form, at the sizes where they can
go wrong: grids of one patch, sizes that no tile divides, stencils of every
window width, items of one source and tiles of many items, sources that share a
stencil origin, grids of very different magnitude, and the line to the direct
kernels; the same for the targets.

Tolerance: 1e-13, as for the integer spread.  The digit sums drop 2^-56 of the
largest coefficient per source and round once per item at the grid's unit;
both, summed over a node's sources, are below the float-float FFT's 2^-48.  The
gather's digits drop 2^-54 of the largest grid value per node."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.fixture(scope="module")
def ft():
    import fasttools2d_gb300 as ft
    return ft


@pytest.fixture(scope="module")
def plans(ft):
    tc, nat = ft.Plan(0), ft.Plan(0)
    nat.set_precision("fp64_native")
    yield tc, nat
    tc.close()
    nat.close()


def _cloud(N, seed, nt=500, Ly=1.0):
    rng = np.random.default_rng(seed)
    box = np.array([[1.0], [Ly]])
    p, q = (rng.random((2, N)) - 0.5) * box, (rng.random((2, nt)) - 0.5) * box
    th = rng.random(N) * 2 * np.pi
    return p, q, rng.standard_normal((2, N)), np.vstack([np.cos(th), np.sin(th)])


def _both(ft, plans, p, q, f, n, Mx, My, P, Ly=1.0, eta=0.9):
    h = 1.0 / Mx
    w = h * P / 2
    xi = 0.95 * np.sqrt(np.pi * P) * np.sqrt(eta) / (2 * w)
    for fn, args in ((ft.mex_stokes_slp_kspace, (f,)), (ft.mex_stokes_dlp_kspace, (f, n))):
        a, b = (fn(p, q, xi, eta, *args, Mx, My, 1.0, Ly, w, P, plan=pl) for pl in plans)
        assert np.all(np.isfinite(a))
        assert relerr(a, b) < TOL, (fn.__name__, relerr(a, b))


@pytest.mark.parametrize("Mx,My,P", [(64, 64, 24), (64, 32, 24), (32, 64, 24), (34, 66, 24), (66, 34, 20), (130, 98, 24),
                                     (104, 200, 4), (200, 104, 6), (128, 128, 10), (96, 96, 16),
                                     (122, 90, 18), (256, 64, 26), (192, 192, 22)])
@pytest.mark.parametrize("N", [1, 17, 4001])
def test_spread_sizes(ft, plans, Mx, My, P, N):
    p, q, f, n = _cloud(N, Mx + My + P + N, Ly=My / Mx)
    _both(ft, plans, p, q, f, n, Mx, My, P, Ly=My / Mx)


@pytest.mark.parametrize("N", [32, 33, 64, 65, 129, 6000])
def test_spread_tiles_of_many_items(ft, plans, N):
    """Sources within one grid cell share every stencil node: items at and around
    their largest size, and tiles of many of them."""
    p, q, f, n = _cloud(N, N)
    p = 0.1 + p / 192
    _both(ft, plans, p, q, f, n, 192, 192, 24)


def test_spread_edges_and_nodes(ft, plans):
    """Sources on nodes, half way between them, and at the ends of the box."""
    M = 128
    e = np.array([-0.5, -0.5 + 1e-15, 0.0, 0.5 / M, 1.0 / M, 0.25, 0.5 - 1.0 / M, 0.5 - 1e-15,
                  3.0 / M + 1e-14, 3.0 / M - 1e-14, 0.49])
    p = np.array([(x, y) for x in e for y in e]).T.copy()
    _, q, f, n = _cloud(p.shape[1], 5)
    _both(ft, plans, p, q, f, n, M, M, 24)


def test_spread_coefficient_range(ft, plans):
    """Coefficients over 16 decades, zeros, and one grid 10^6 times another."""
    p, q, f, n = _cloud(20000, 9)
    rng = np.random.default_rng(10)
    g = f * 10.0 ** rng.uniform(-8, 8, f.shape[1])
    g[:, ::7] = 0.0
    _both(ft, plans, p, q, g, n, 192, 192, 24)
    g = f.copy()
    g[1] *= 1e-6
    _both(ft, plans, p, q, g, n, 192, 192, 24)
    g[1] = 0.0
    _both(ft, plans, p, q, g, n, 192, 192, 24)


@pytest.mark.parametrize("M", [512, 896, 1344, 2688])
def test_spread_either_side_of_the_sparse_line(ft, plans, M):
    """8000 sources: dense enough for tiles up to 896^2 nodes, the direct spread beyond."""
    p, q, f, n = _cloud(8000, M)
    _both(ft, plans, p, q, f, n, M, M, 24)


def test_spread_tiles_of_many_items_are_reproducible(ft, plans):
    """Tiles of many items: the same bits on every call."""
    rng = np.random.default_rng(3)
    p, q, f, n = _cloud(20000, 3)
    p = (0.3 * rng.standard_normal((2, 20000)) + 0.5) % 1.0 - 0.5
    a = [ft.mex_stokes_dlp_kspace(p, q, 60.0, 0.85, f, n, 192, 192, 1.0, 1.0, 12 / 192, 24,
                                  plan=plans[0]) for _ in range(3)]
    assert np.array_equal(a[0], a[1]) and np.array_equal(a[0], a[2])


@pytest.mark.parametrize("nt", [1, 31, 33, 64, 65, 3000])
def test_gather_items(ft, plans, nt):
    """Targets over the box, and all in one grid cell (a tile of many items)."""
    p, q, f, n = _cloud(3000, 60 + nt, nt=nt)
    _both(ft, plans, p, q, f, n, 192, 192, 24)
    _both(ft, plans, p, -0.2 + q / 192, f, n, 192, 192, 24)


def test_gather_edges_and_nodes(ft, plans):
    M = 128
    e = np.array([-0.5, -0.5 + 1e-15, 0.0, 0.5 / M, 1.0 / M, 0.25, 0.5 - 1.0 / M, 0.5 - 1e-15,
                  3.0 / M + 1e-14, 3.0 / M - 1e-14, 0.49])
    q = np.array([(x, y) for x in e for y in e]).T.copy()
    p, _, f, n = _cloud(2000, 7)
    _both(ft, plans, p, q, f, n, M, M, 24)


@pytest.mark.parametrize("M", [512, 1344, 2688])
def test_gather_either_side_of_the_sparse_line(ft, plans, M):
    p, q, f, n = _cloud(500, M, nt=65536)
    _both(ft, plans, p, q, f, n, M, M, 24)


@pytest.mark.parametrize("M,P,N,xi,nside", [(64, 24, 40, 20.0, 4), (96, 24, 1500, 30.0, 6), (98, 20, 65, 30.0, 6),
                                            (130, 10, 700, 40.0, 8), (192, 26, 3000, 55.0, 11)])
def test_adjoint_gather(ft, plans, M, P, N, xi, nside):
    """Gradients of the tensor-core adjoint gather against the all-FP64 form, at the
    1e-11 of the float-float adjoint's test."""
    rng = np.random.default_rng(M + N)
    p, q, f, n = _cloud(N, M, nt=300)
    g, w1, w2 = rng.standard_normal((2, N)), rng.standard_normal((2, 300)), rng.standard_normal((2, 300))
    p[:, : N // 4] = 0.05 + p[:, : N // 4] / M       # one grid cell: a tile of many items
    prm = ft.EwaldParams.derived(xi, nside, nside, M, M, P, 1.0, 1.0)
    a, b = (ft.stokes_ewald_adjoint(p, q, f, g, n, w1, w2, prm, plan=pl) for pl in plans)
    for x, y in zip(a, b):
        assert relerr(x, y) < 1e-11, relerr(x, y)
