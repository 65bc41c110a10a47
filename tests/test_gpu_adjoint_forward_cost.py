"""LiftObjective.forward keeps the last segment's stages for a reverse sweep that may never come (a line search
evaluates forward alone): a run whose last segment is all of it takes no longer than one that keeps a single
step of the same 40."""
import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(64, 16), (256, 64)])
def test_keeping_the_stages_costs_a_forward_run_nothing(pkg, size):
    mesh = pkg.Mesh.naca_ogrid(*size, farfield="characteristic")
    objs = [pkg.LiftObjective(mesh, pkg.config(N=3, cfl=0.5, mach=0.4, alpha_deg=1.0), 40, 1, C) for C in (39, 40)]
    best = [1e9, 1e9]
    for _ in range(20):  # in turn; the best of each
        for k, o in enumerate(objs):
            t = time.perf_counter()
            o.forward()
            best[k] = min(best[k], time.perf_counter() - t)
    # one step against 40 kept: 27 % (K = 2048) and 7 % (K = 32768) apart with a copy after each stage
    assert best[1] < 1.04 * best[0], best
