"""The advection right-hand side conserves: what leaves a cell through a face enters its neighbour.  Each side of a
face forms its own flux in the fused stage kernel, so the pair cancels to rounding, as in the forms with one
flux per face (whose sides scale it by their own fscale)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("n", [20, 79])  # both block sizes
def test_right_hand_side_integrates_to_zero(pkg, oops, omesh, N, n):
    """The integral of the right-hand side over the domain, with the ghost value on and near the boundary (whose
    fluxes then cancel around it) and O(1) noise inside.  Every cell's integral is a sum of about a hundred products
    of size 1 / h, each rounded to 2^-53, and 2 n^2 cells of either sign add at random: 1e-13 of the sum of
    the magnitudes is some ten times that."""
    op = oops.operators(N)
    r, s = np.asarray(op["r"]), np.asarray(op["s"])
    V = oops.vandermonde_2d(N, r, s)
    w = np.linalg.inv(V @ V.T).sum(axis=1)  # integrals of the nodal basis over the reference triangle
    assert abs(w.sum() - 2.0) < 1e-12
    m = omesh.vortex_square(n, 0.0, 1.0)
    c = m["coords"][m["cell2nodes"]]  # [cell][vertex][2]
    inside = ((c > 2.5 / n) & (c < 1 - 2.5 / n)).all(axis=(1, 2))
    rng = np.random.default_rng(N)
    q = np.full((len(c), w.size), 4.5e-5)
    q[inside] += rng.uniform(-1, 1, (int(inside.sum()), w.size))
    area = 0.5 * abs((c[:, 1, 0] - c[:, 0, 0]) * (c[:, 2, 1] - c[:, 0, 1]) - (c[:, 2, 0] - c[:, 0, 0]) * (c[:, 1, 1] - c[:, 0, 1]))
    mesh = pkg.Mesh.from_tables(m)
    for form in (0, 3):
        pkg.lib().dg_set_elem_variant(form)
        try:
            a = pkg.Advection(mesh, N=N, vel_x=0.9, vel_y=-0.4, dt=1e-3).init()
            rhs = a.rhs(q.ravel()).reshape(q.shape)
        finally:
            pkg.lib().dg_set_elem_variant(3)
        per_node = rhs * w * (area / 2)[:, None]
        assert abs(per_node.sum()) < 1e-13 * abs(per_node).sum(), form
