"""Real-space sums over many runs per block, against the same points alone.

The real-space kernels cut their outer points into runs that blocks take as they
get free; a point's sum depends neither on the other points nor on the block.  The
points here crowd around an arc, so that a warp has several runs, and a few of them
evaluated alone (one point per warp) must give the same sums to rounding: a sum of
at most 3001 terms in float-float (2^-47 each) and FP64 stays within 1e-12 of the
largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def ft():
    import fasttools2d_gb300 as ft
    return ft


def _arc(rng, n):
    th = rng.random(n) * 2.5
    r = 0.3 + 0.02 * rng.standard_normal(n)
    return np.vstack([r * np.cos(th), r * np.sin(th)])


@pytest.mark.parametrize("precision", ["fp64", "fp64_native", "fp32_grid"])
@pytest.mark.parametrize("n", [30011, 14592])
def test_sums_do_not_depend_on_the_runs(ft, precision, n):
    rng = np.random.default_rng(n)
    ps, pt = _arc(rng, 3001), _arc(rng, n)
    pt[:, :50] = ps[:, :50]
    f, g = rng.standard_normal((2, 3001)), rng.standard_normal((2, 3001))
    few = np.sort(rng.choice(n, 200, replace=False))
    plan = ft.Plan(0)
    try:
        plan.set_precision(precision)
        for run in (lambda t: ft.mex_stokes_slp_real(ps, t, f, 18.0, 3, 3, 1.0, 1.0, plan=plan),
                    lambda t: ft.mex_stokes_dlp_real(ps, t, f, g, 18.0, 3, 3, 1.0, 1.0, plan=plan)):
            u = run(pt)
            alone = run(np.ascontiguousarray(pt[:, few]))
            tol = 1e-5 if precision == "fp32_grid" else TOL   # (far pairs in FP32 there)
            assert np.abs(u[:, few] - alone).max() <= tol * np.abs(u).max()
    finally:
        plan.close()


@pytest.mark.parametrize("precision", ["fp64", "fp64_native"])
def test_gradients_do_not_depend_on_the_runs(ft, precision):
    rng = np.random.default_rng(5)
    n = 30011
    ps, pt = _arc(rng, n) + 0.5, _arc(rng, 3001) + 0.5
    f, g, nr = (rng.standard_normal((2, n)) for _ in range(3))
    w1, w2 = rng.standard_normal((2, 3001)), rng.standard_normal((2, 3001))
    few = np.sort(rng.choice(n, 200, replace=False))
    prm = ft.EwaldParams.derived(18.0, 3, 3, 64, 64, 20, 1.0, 1.0)
    plan = ft.Plan(0)
    try:
        plan.set_precision(precision)
        grads = ft.stokes_ewald_adjoint(ps, pt, f, g, nr, w1, w2, prm, plan=plan)
        cut = [np.ascontiguousarray(x[:, few]) for x in (ps, f, g, nr)]
        alone = ft.stokes_ewald_adjoint(cut[0], pt, *cut[1:], w1, w2, prm, plan=plan)
        for a, b in zip(grads, alone):
            assert np.abs(a[:, few] - b).max() <= TOL * np.abs(a).max()
    finally:
        plan.close()


@pytest.mark.parametrize("far", [3.0e4, 1.5e7])
@pytest.mark.parametrize("box", [(1.0, 1.0, 1, 1), (1.0, 2.0, 1, 2)])
def test_pairs_far_outside_the_cell(ft, far, box):
    """All points far outside the cell (the reference puts them into one edge box), where
    the FP32 pre-test of the cutoff cannot decide for their images: the oracle's pair set
    and sums (1e-12, as the other comparisons with it: the same FP64 offsets, then at
    most 400 terms).  In FP64 throughout: the float-float form takes its pairs by the
    FP32 distance, which has no digits left there."""
    from oracle import oracle as O
    Lx, Ly, nx, ny = box
    rng = np.random.default_rng(int(far) + ny)
    ps, pt = (np.vstack([far + (rng.random(400) - 0.5) * Lx, (rng.random(400) - 0.5) * Ly - far])
              for _ in range(2))
    f, g = rng.standard_normal((2, 400)), rng.standard_normal((2, 400))
    xi = 3.0 * max(nx / Lx, ny / Ly)
    plan = ft.Plan(0)
    try:
        plan.set_precision("fp64_native")
        for got, ref in ((ft.mex_stokes_slp_real(ps, pt, f, xi, nx, ny, Lx, Ly, plan=plan),
                          O.mex_stokes_slp_real(ps, pt, f, xi, nx, ny, Lx, Ly)),
                         (ft.mex_stokes_dlp_real(ps, pt, f, g, xi, nx, ny, Lx, Ly, plan=plan),
                          O.mex_stokes_dlp_real(ps, pt, f, g, xi, nx, ny, Lx, Ly))):
            assert np.isfinite(ref).all()
            assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    finally:
        plan.close()
