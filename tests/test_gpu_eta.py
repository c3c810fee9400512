"""The k space over the spectral splitting parameter eta, which callers choose freely: the
Gaussians' exponent per node spacing, alpha = 2 xi^2 h^2 / eta, on both sides of the
lines beyond which the tensor-core spread and gather leave the call to the integer
kernels, against the all-FP64 form.

Tolerance: 1e-13 as for the other k-space tests, but no less than 12 alpha P 2^-53: the
FP64 form takes each Gaussian factor as a product of exponentials of up to alpha P, each
off by its exponent times 2^-53 (three of them, two axes, spread and gather).  Gradients:
1e-11, as in the adjoint's other tests."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


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


def _tol(alpha, P):
    return max(1e-13, 12 * alpha * P * 2.0 ** -53)


def _cloud(N, nt, seed):
    rng = np.random.default_rng(seed)
    p, q = rng.random((2, N)) - 0.5, rng.random((2, nt)) - 0.5
    th = rng.random(N) * 2 * np.pi
    # of one sign and smooth: neighbouring nodes all near the grid's maximum
    f = np.vstack([1 + 0.3 * np.cos(2 * np.pi * p[0]), 1 + 0.2 * np.sin(2 * np.pi * p[1])])
    return p, q, f, np.vstack([np.cos(th), np.sin(th)])


def _kspace(ft, plans, M, P, xi, eta):
    p, q, f, n = _cloud(2000, 2000, P)
    h = 1.0 / M
    for fn, args in ((ft.mex_stokes_slp_kspace, (f,)), (ft.mex_stokes_dlp_kspace, (f, n))):
        a, b = (fn(p, q, xi, eta, *args, M, M, 1.0, 1.0, h * P / 2, P, plan=pl) for pl in plans)
        err = relerr(a, b)
        assert err < _tol(2 * xi * xi * h * h / eta, P), (fn.__name__, err)


def _gradients(ft, plans, M, P, xi, eta):
    p, q, f, n = _cloud(2000, 2000, P)
    prm = ft.EwaldParams(xi, 4, 4, M, M, P, 1.0, 1.0, P / M / 2, eta)
    a, b = (ft.stokes_ewald_adjoint(p, q, f, f, n, 1 + 0 * q, 1 + 0 * q, prm, plan=pl) for pl in plans)
    for x, y in zip(a, b):
        assert relerr(x, y) < 1e-11, relerr(x, y)


@pytest.mark.parametrize("P,alpha", [(4, 10.9), (4, 11.2), (4, 25.0), (8, 11.2), (8, 35.0), (16, 11.2), (16, 17.0),
                                     (24, 10.9), (24, 11.2), (24, 12.0)])
def test_narrow_gaussians(ft, plans, P, alpha):
    M = 256
    xi = 0.4 * M / P
    eta = 2 * xi * xi / (M * M) / alpha
    _kspace(ft, plans, M, P, xi, eta)
    _gradients(ft, plans, M, P, xi, eta)


FLAT = [0.3, 1.0, 1.2, 1.5, 2.0, 2.4, 2.6, 3.0, 4.0, 6.0, 8.0]


@pytest.mark.parametrize("P", [4, 12, 24, 26])
@pytest.mark.parametrize("ratio", FLAT)
def test_flat_gaussians(ft, plans, P, ratio):
    """eta at multiples of the drivers' choice (which is 0.05 here, so that the filter
    does not amplify the rounding of either side)."""
    M = 256
    xi = 0.95 * np.sqrt(np.pi * P) * np.sqrt(0.05) / (P / M)
    _kspace(ft, plans, M, P, xi, 0.05 * ratio)
    _gradients(ft, plans, M, P, xi, 0.05 * ratio)
