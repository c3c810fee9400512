"""Waits of the tensor-core kernels that run out: the call reports it, and the plan goes on.

With a limit of 0 polls every wait gives up before it looks, with 1 some do on the way,
with products, bulk reductions and other blocks in flight."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ft():
    import fasttools2d_gb300 as ft
    return ft


def _cloud(N, seed):
    rng = np.random.default_rng(seed)
    p, q = rng.random((2, N)) - 0.5, rng.random((2, N)) - 0.5
    th = rng.random(N) * 2 * np.pi
    return p, q, rng.standard_normal((2, N)), np.vstack([np.cos(th), np.sin(th)])


def _call(ft, plan, op, N):
    p, q, f, n = _cloud(N, 3)
    prm = ft.EwaldParams.derived(60.0, 12, 12, 192, 192, 24, 1.0, 1.0)
    if op == "slp":
        return (ft.slp_ewald(p, q, f, prm, plan=plan),)
    if op == "stokes":
        return ft.stokes_ewald(p, q, f, f, n, prm, plan=plan)
    if op == "adjoint":
        return ft.stokes_ewald_adjoint(p, q, f, f, n, f, f, prm, plan=plan)
    geo = ft.Geometry(p, q, prm, n=n, plan=plan)
    try:
        return geo.apply(np.stack([f, 2 * f]), np.stack([f, 2 * f]))
    finally:
        geo.close()


@pytest.mark.parametrize("N", [500, 40000])
@pytest.mark.parametrize("op", ["slp", "stokes", "adjoint", "geometry"])
def test_a_wait_that_runs_out(ft, op, N):
    plan = ft.Plan(0)
    want = _call(ft, plan, op, N)
    for polls in (0, 1, 0):
        plan.set_wait_limit(polls)
        try:
            got = _call(ft, plan, op, N)
            assert polls > 0                         # (it may have been fast enough)
            assert all(relerr(x, y) < 1e-11 for x, y in zip(got, want))
        except ft.Se2pError as e:
            assert e.code == 2 and "tensor-core" in str(e)
        plan.set_wait_limit()
        got = _call(ft, plan, op, N)
        assert all(relerr(x, y) < 1e-11 for x, y in zip(got, want))
    plan.close()


@pytest.mark.parametrize("op", ["slp", "adjoint"])
def test_queued_calls(ft, op):
    """On CUDA tensors the call has returned before its kernels run: its results are NaN,
    and the plan's synchronize or its next call reports it, once."""
    import torch
    p, q, f, n = (torch.tensor(np.ascontiguousarray(x.T), device="cuda") for x in _cloud(5000, 8))
    prm = ft.EwaldParams.derived(60.0, 12, 12, 192, 192, 24, 1.0, 1.0)
    plan = ft.Plan(0)

    def call():
        if op == "slp":
            return ft.slp_ewald(p, q, f, prm, parts=True, plan=plan)
        return ft.stokes_ewald_adjoint(p, q, f, f, n, f, f, prm, plan=plan)

    want = call()
    plan.synchronize()
    for ask in (plan.synchronize, call):
        plan.set_wait_limit(0)
        got = call()
        torch.cuda.synchronize()
        if op == "slp":
            assert torch.isnan(got[0]).all() and torch.isnan(got[2]).all()
            assert (got[1] - want[1]).abs().max() <= 1e-12 * want[1].abs().max()
        else:
            assert all(torch.isnan(g).all() for g in got)
        plan.set_wait_limit()
        with pytest.raises(ft.Se2pError, match="tensor-core"):
            ask()
        got = call()
        plan.synchronize()
        for x, y in zip(got, want):
            assert relerr(x.cpu().numpy(), y.cpu().numpy()) < 1e-11
    plan.close()


def test_limits(ft):
    plan = ft.Plan(0)
    for bad in (-1, (1 << 16) + 1):
        with pytest.raises(ft.Se2pError):
            plan.set_wait_limit(bad)
    plan.close()
