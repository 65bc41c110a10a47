"""The batch's grouped launches on both sides of the small-tile rule, which there goes by the cells of all
instances of an order: with few of them small tiles, with many 32-cell tiles, while each instance alone is
small enough for small tiles in its own solver.  Bit for bit the same either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# order: instances whose cells are below the solver's line for small tiles and together above the batch's
# (at order 5 the lines are bands: 8,193 to 9,728 cells together, 5,120 or fewer each, of which 2,433 to
# 4,864 have 32-cell tiles alone too)
SIZES = {1: [(64, 96)] * 3, 3: [(64, 80)] * 2 + [(47, 41)], 4: [(64, 40)] * 2, 5: [(32, 80), (31, 70)]}


@pytest.mark.parametrize("shape", [None, (99, 64), (99, 256)])
@pytest.mark.parametrize("N", [1, 3, 4, 5])
def test_grouped_32_cell_tiles_equal_the_plain_solvers(pkg, N, shape):
    total = sum(2 * a * b for a, b in SIZES[N])
    assert total > {1: 32768, 3: 20480, 4: 8192, 5: 8192}[N] and (N != 5 or total <= 9728)
    meshes = [pkg.Mesh.naca_ogrid(*s) for s in SIZES[N]]
    cfgs = [pkg.config(N=N, cfl=0.3, mach=0.4 + 0.02 * k, alpha_deg=k) for k in range(len(meshes))]
    b = pkg.Batch(meshes, cfgs).init()
    if shape:
        b.use_shape(*shape)
    b.run(10)  # the eight-step graph and two single steps
    b.sync()
    for k, (m, c) in enumerate(zip(meshes, cfgs)):
        s = pkg.Solver(m, c).init()
        s.run(10)
        s.sync()
        assert np.array_equal(s.get("q"), b.get(k)) and s.time() == b.time(k)


def test_tiles_follow_a_change_of_shape_with_steps_in_flight(pkg):
    """use_shape replaces the tiles that the graphs of earlier steps hold, without a wait in between."""
    meshes = [pkg.Mesh.naca_ogrid(*s) for s in ((47, 11), (33, 7), (64, 40))]
    cfgs = [pkg.config(N=n, cfl=0.3, mach=0.5, alpha_deg=1.0) for n in (3, 2, 4)]
    b = pkg.Batch(meshes, cfgs).init()
    for shape in ((99, 64), (2, 1024), (99, 128), (2, 2048), (99, 64)):
        b.use_shape(*shape)
        b.run(9)
    b.sync()
    for k, (m, c) in enumerate(zip(meshes, cfgs)):
        s = pkg.Solver(m, c).init()
        s.run(45)
        s.sync()
        assert np.array_equal(s.get("q"), b.get(k)) and s.time() == b.time(k)
