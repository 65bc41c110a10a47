"""The reverse sweep starts with the stages that the forward run kept of its last segment; a call in
between that moves the solver's state or uses the segment buffers (rhs_vjp, tangent), or an earlier
reverse sweep over several segments, makes it recompute them.  Both ways compute the same bits, and
leave the same step state behind (rhs_vjp's boundary time in the vortex app)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def objective(pkg, app, nsteps, C):
    if app:
        mesh = pkg.Mesh.vortex_square(8, -5.0, 5.0)
        cfg = pkg.config(N=3, cfl=0.5, app=1, vortex_x0=0.3, vortex_y0=0.1)
        return mesh, cfg, pkg.LiftObjective(mesh, cfg, nsteps, 1, C)
    mesh = pkg.Mesh.naca_ogrid(32, 8, radius=4.0, farfield="characteristic")
    cfg = pkg.config(N=3, cfl=0.5, mach=0.5, alpha_deg=2.0)
    return mesh, cfg, pkg.LiftObjective(mesh, cfg, nsteps, min(3, nsteps), C)


# one segment, exactly full segments, a short last one of one step, several steps
@pytest.mark.parametrize("nsteps,C", [(5, 9), (6, 3), (7, 3), (8, 3), (1, 1)])
@pytest.mark.parametrize("app", [0, 1])
def test_kept_stages_equal_recomputed(pkg, app, nsteps, C):
    mesh, cfg, obj = objective(pkg, app, nsteps, C)
    q = pkg.Solver(mesh, cfg).init().get("q")
    v = np.random.default_rng(3).standard_normal(q.size)
    J = obj.forward()
    kept = obj.backward()
    after = obj.rhs_vjp(q, v)  # with the step state that the sweep left; uses the segment buffers
    for between in ("vjp", "tangent", "sweep"):
        if between == "tangent":
            assert obj.forward() == J
            obj.tangent(1.0)
        elif between == "sweep":
            assert obj.forward() == J
            obj.backward()
        again = obj.backward()
        assert again[0] == kept[0] and np.array_equal(again[1], kept[1]), between
        av = obj.rhs_vjp(q, v)
        assert np.array_equal(av[0], after[0]) and av[1] == after[1], between
