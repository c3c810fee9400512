"""Plans of different grids and stencils in several threads at once: each call's results
are those of the same call alone."""
import threading

import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


def test_threads_with_different_sizes():
    import fasttools2d_gb300 as ft
    failed = []

    def work(P, M, seed):
        try:
            rng = np.random.default_rng(seed)
            p, q, f = (rng.random((2, n)) - 0.5 for n in (2000, 500, 2000))
            xi = 0.9 * np.sqrt(np.pi * P) / (P / M)
            plan = ft.Plan(0)
            first = None
            for _ in range(200):
                u = ft.mex_stokes_slp_kspace(p, q, xi, 0.9, f, M, M, 1.0, 1.0, P / M / 2, P, plan=plan)
                first = u if first is None else first
                assert relerr(u, first) < 1e-13
            plan.close()
        except Exception as e:
            failed.append((P, M, repr(e)))

    threads = [threading.Thread(target=work, args=a) for a in
               ((26, 640, 1), (4, 104, 2), (12, 128, 3), (24, 96, 4))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
