"""Few points on a fine grid: the integer spread and gather and the float-float adjoint
gather, alone and for batches of densities, which the tensor-core kernels leave such calls
to.  Against the all-FP64 form; tolerances as in the tests of the same entry points
(adjoint 1e-11, potentials 1e-12, a batch against single evaluations 3e-13)."""
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
    a, nat = ft.Plan(0), ft.Plan(0)
    nat.set_precision("fp64_native")
    yield a, nat
    a.close()
    nat.close()


def _cloud(N, seed):
    rng = np.random.default_rng(seed)
    p, q = rng.random((2, N)) - 0.5, rng.random((2, N)) - 0.5
    th = rng.random(N) * 2 * np.pi
    return p, q, np.vstack([np.cos(th), np.sin(th)]), rng.standard_normal((3, 2, N))


@pytest.mark.parametrize("kind", ["both", "slp", "dlp"])
@pytest.mark.parametrize("M,P", [(1344, 24), (2688, 12), (1344, 26)])
def test_adjoint(ft, plans, kind, M, P):
    N = 8000
    p, q, n, f = _cloud(N, M + P)
    prm = ft.EwaldParams.derived(M / 3.15, 85, 85, M, M, P, 1.0, 1.0)
    fs, ws = (f[0], f[1]) if kind != "dlp" else (None, None)
    fd, wd = (f[2], f[1]) if kind != "slp" else (None, None)
    a, b = (ft.stokes_ewald_adjoint(p, q, fs, fd, n if kind != "slp" else None, ws, wd, prm, plan=pl)
            for pl in plans)
    for x, y in zip(a, b):
        assert (x is None) == (y is None)
        assert x is None or relerr(x, y) < 1e-11, relerr(x, y)


@pytest.mark.parametrize("kinds", ["both", "slp", "dlp"])
@pytest.mark.parametrize("bad", [None, 0, 1])
def test_batch(ft, plans, kinds, bad):
    N, M = 8000, 1792
    p, q, n, f = _cloud(N, M)
    if bad is not None:
        f[bad, 1, 77] = np.nan
    prm = ft.EwaldParams.derived(M / 3.15, 110, 110, M, M, 24, 1.0, 1.0)
    geo = ft.Geometry(p, q, prm, n=None if kinds == "slp" else n, kinds=kinds, plan=plans[0])
    us, ud = geo.apply(f if kinds != "dlp" else None, f if kinds != "slp" else None)
    for r in range(3):
        single = []
        for pl in plans:
            if kinds == "both":
                single.append(ft.stokes_ewald(p, q, f[r], f[r], n, prm, plan=pl))
            elif kinds == "slp":
                single.append((ft.slp_ewald(p, q, f[r], prm, plan=pl), None))
            else:
                single.append((None, ft.dlp_ewald(p, q, f[r], n, prm, plan=pl)))
        for u, v, w in zip((us, ud), *single):
            if u is None:
                continue
            assert np.array_equal(np.isfinite(u[r]), np.isfinite(v))
            if r != bad:
                assert np.isfinite(u[r]).all()
                assert relerr(u[r], v) < 3e-13 and relerr(u[r], w) < 1e-12, (relerr(u[r], v), relerr(u[r], w))
    geo.close()
