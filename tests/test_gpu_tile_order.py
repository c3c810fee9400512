"""Tiles of very many sources: the order of their items, on both sides of the lines beyond
which one block orders a tile (2^16 sources, 4096 of them in the tile), against the all-FP64 form (1e-13, as for the other k-space
tests) and against the same call again (bit for bit: each item holds the same sources on
every call, whatever order the atomics found)."""
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


def _check(ft, plans, p, f, M=128, P=24):
    q = np.random.default_rng(1).random((2, 400)) - 0.5
    xi = 0.9 * np.sqrt(np.pi * P) / (P / M)
    a, a2, b = (ft.mex_stokes_slp_kspace(p, q, xi, 0.9, f, M, M, 1.0, 1.0, P / M / 2, P, plan=pl)
                for pl in (plans[0], plans[0], plans[1]))
    assert np.array_equal(a, a2)
    assert relerr(a, b) < 1e-13, relerr(a, b)


@pytest.mark.parametrize("others", [0, 62000])
@pytest.mark.parametrize("N", [4095, 4096, 4097, 4352, 16000])
def test_one_tile(ft, plans, N, others):
    """One tile of N, the other sources spread over the cell (about 1300 to a tile)."""
    rng = np.random.default_rng(N + others)
    p = np.concatenate([0.1 + rng.random((2, N)) / 128, rng.random((2, others)) - 0.5], 1)
    p = p[:, rng.permutation(N + others)]
    f = rng.standard_normal(p.shape)
    f[:, rng.random(N + others) < 0.5] = 0.0         # (half of them: below the crowding line)
    _check(ft, plans, p, f)


@pytest.mark.parametrize("N,at", [(65536, "spread"), (65537, "first"), (65537, "spread"), (200000, "spread")])
def test_few_densities_on_many_sources(ft, plans, N, at):
    """(sources without a density do not count as crowded)"""
    rng = np.random.default_rng(N)
    f = rng.standard_normal((2, N))
    f[:, (np.arange(N) >= 500) if at == "first" else (np.arange(N) % 97 != 0)] = 0.0
    _check(ft, plans, 0.1 + rng.random((2, N)) / 128, f)


@pytest.mark.parametrize("numbering", ["in turn", "runs", "outlier", "shuffled"])
def test_several_tiles(ft, plans, numbering):
    """Two long tiles and a background of short ones, whose sources the caller numbers in
    turn, tile by tile, with one number far from the others, or at random."""
    rng = np.random.default_rng(9)
    n = 31000
    c = [x + rng.random((2, n)) / 128 for x in (-0.3, 0.2)]
    bg = rng.random((2, 5000)) - 0.5
    if numbering == "in turn":
        p = np.concatenate([np.stack(c, 2).reshape(2, 2 * n), bg], 1)
    elif numbering == "runs":
        p = np.concatenate([c[0], bg, c[1]], 1)
    elif numbering == "outlier":
        p = np.concatenate([c[0][:, :1], bg, c[1], c[0][:, 1:]], 1)
    else:
        p = np.concatenate([c[0], bg, c[1]], 1)[:, rng.permutation(2 * n + 5000)]
    f = rng.standard_normal(p.shape)
    f[:, rng.random(f.shape[1]) < 0.7] = 0.0         # (below the crowding line)
    _check(ft, plans, p, f)
    _check(ft, plans, p, f, M=64, P=4)
