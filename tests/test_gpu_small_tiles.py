"""Small element tiles (8 or 16 cells) of the tensor-core forms against the 32-cell tiles, over sizes that
are not multiples of either, and against the oracle where the other forms' sums differ (N = 1, 2, 6)."""
import numpy as np
import pytest

from conftest import push_affine_geometry

pytestmark = pytest.mark.gpu


def _steps(pkg, mesh, cfg, variant, steps):
    pkg.lib().dg_set_elem_variant(variant)
    try:
        s = pkg.Solver(mesh, cfg).init()
        s.record_dt(steps)
        s.run(steps)
        s.sync()
        W = s.get("q") * 1.01
        return s.get("q"), s.dt_history(steps), s.rhs(W)
    finally:
        pkg.lib().dg_set_elem_variant(3)


@pytest.mark.parametrize("N", [3, 4, 5])
@pytest.mark.parametrize("size", [(9, 1), (8, 2), (33, 7), (47, 41), (64, 64)])
def test_small_tiles_equal_32_cell_tiles(pkg, N, size):
    """Form 2 runs 32-cell tiles with the same contraction: q, dt and one right-hand side bit for bit
    (a column's operands and exponent do not depend on the tile it is in)."""
    mesh = pkg.Mesh.naca_ogrid(*size)
    cfg = pkg.config(N=N, cfl=0.3, mach=0.5, alpha_deg=2.0)
    small, ref = _steps(pkg, mesh, cfg, 3, 11), _steps(pkg, mesh, cfg, 2, 11)
    for a, b in zip(small, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("N", [1, 2, 6])
@pytest.mark.parametrize("size", [(8, 1), (9, 1), (33, 7), (47, 41)])
def test_small_tiles_match_oracle(pkg, orc, oops, omesh, N, size):
    """The tensor-core forms at N = 1, 2 (dense) and 6 (even/odd, three k-steps) on tiles of 8 and 16
    cells: one right-hand side of a
    state with 5 % noise to 1e-13, as the other right-hand-side tests."""
    m = omesh.naca_ogrid(*size, farfield="characteristic")
    s = pkg.Solver(pkg.Mesh.from_tables(m), pkg.config(N=N, cfl=0.5)).init()
    o = orc.Oracle(m, oops.operators(N), orc.freestream(0.4, 0.0), kind="port")
    o.init(0.5)
    push_affine_geometry(o, s.get("geo").reshape(-1, 16))
    q = o.get("q")
    W = q * (1.0 + 0.05 * np.random.default_rng(N).standard_normal(q.size))
    o.set("workingQ", W)
    assert orc.rel_l2(s.rhs(W), o.rhs(0)) < 1e-13


@pytest.mark.parametrize("N", [1, 2, 6])
@pytest.mark.parametrize("variant", [2, 99])
def test_batch_equals_small_tiles(pkg, N, variant):
    """The batch's 32-cell tiles (persistent and grouped launches) give each instance what its own
    solver's small tiles give, bit for bit."""
    meshes = [pkg.Mesh.naca_ogrid(*size) for size in ((9, 1), (47, 11))]
    cfgs = [pkg.config(N=N, cfl=0.3, mach=0.5, alpha_deg=a) for a in (0.0, 2.0)]
    b = pkg.Batch(meshes, cfgs).init()
    b.use_shape(variant, 64)
    b.run(7)
    b.sync()
    for k, (m, c) in enumerate(zip(meshes, cfgs)):
        s = pkg.Solver(m, c).init()
        s.run(7)
        s.sync()
        assert np.array_equal(s.get("q"), b.get(k)) and s.time() == b.time(k)
