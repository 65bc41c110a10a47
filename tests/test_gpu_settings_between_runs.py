"""A solver's step graphs (one step, several, with host copies) are captured when a call first needs each: all
of them under the settings of the first, so that a change of the element form between two runs does not mix
two arithmetics in one solver."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def forms(pkg):
    yield pkg.lib().dg_set_elem_variant
    pkg.lib().dg_set_elem_variant(3)


@pytest.mark.parametrize("other", [0, 1])
@pytest.mark.parametrize("first,second", [(8, 9), (1, 8), (3, 17)])
@pytest.mark.parametrize("size", [(24, 6), (128, 32)])  # one range; two cell ranges
def test_runs_keep_the_first_form(pkg, forms, size, first, second, other):
    mesh, cfg = pkg.Mesh.naca_ogrid(*size), pkg.config(N=3, cfl=0.5, mach=0.4, alpha_deg=2.0)
    want = pkg.Solver(mesh, cfg).init()
    want.run(first + second)
    want.sync()
    s = pkg.Solver(mesh, cfg).init()
    s.run(first)
    forms(other)
    s.run(second)
    s.sync()
    assert np.array_equal(want.get("q"), s.get("q")) and want.time() == s.time()


@pytest.mark.parametrize("first,second", [(8, 9), (1, 8)])
@pytest.mark.parametrize("N", [1, 3, 4])
def test_advection_runs_keep_the_first_form(pkg, forms, N, first, second):
    mesh = pkg.Mesh.vortex_square(9, 0.0, 1.0)
    got = []
    for change in (False, True):
        forms(3)
        a = pkg.Advection(mesh, N=N, vel_x=0.9, vel_y=-0.4, dt=1e-3).init()
        a.run(first)
        if change:
            forms(0)
        a.run(second)
        a.sync()
        got.append(a.get("q"))
    assert np.array_equal(*got)
