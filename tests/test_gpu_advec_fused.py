"""The advection stage kernel (staging, face terms, tensor-core contraction and RK4 combine in one)
against the dense FP64 form (0), over cell counts that fill no tile, both block sizes, and a mesh whose
neighbouring cells are far apart in number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shuffled(m, seed):
    new = np.random.default_rng(seed).permutation(len(m["cell2nodes"])).astype(np.int32)
    out = dict(m)
    c = np.empty_like(m["cell2nodes"])
    c[new] = m["cell2nodes"]
    out.update(cell2nodes=c, edge2cells=new[m["edge2cells"]], bedge2cell=new[m["bedge2cell"]])
    return out


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("n", [1, 3, 7, 20, 79])  # 2 n^2 cells; 128-cell blocks above 12288
def test_fused_stage_equals_dense_form(pkg, orc, omesh, N, n):
    """One right-hand side of a perturbed state and q after five steps, 1e-13 as the forms' other test;
    W holds the new state after a step."""
    m = _shuffled(omesh.vortex_square(n, 0.0, 1.0), n)
    got = []
    for form in (0, 3):
        pkg.lib().dg_set_elem_variant(form)
        try:
            a = pkg.Advection(pkg.Mesh.from_tables(m), N=N, vel_x=0.9, vel_y=-0.4, dt=0.1 / (n * (N + 1) ** 2)).init()
            q = a.get("q")
            r = a.rhs(q + 0.5 * np.random.default_rng(N).uniform(-1, 1, q.size))
            a.set("workingQ", q)
            a.run(5)
            a.sync()
            assert np.array_equal(a.get("q"), a.get("workingQ"))
            a.run(9)  # the eight-step graph and a single step
            a.sync()
            got.append((r, a.get("q")))
        finally:
            pkg.lib().dg_set_elem_variant(3)
    for x, y in zip(*got):
        assert orc.rel_l2(y, x) < 1e-13
