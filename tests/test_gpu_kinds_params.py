"""k_assemble_kinds after new spring parameters, on cloths whose springs of a kind differ in their
rest lengths by their place in the grid (parameter slots, not a rest length per spring): the rest
lengths stay each spring's own, whether the kind shared one Ks when the handle was made or only
after oc_set_spring_params."""
import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, grid_cloth, ClothSolver
from test_gpu_kinds import run

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def cloth(cols, rows, ks_edge):
    """The reference's lattice; the first row's horizontal springs are shorter, and of Ks ks_edge."""
    X, sp = grid_cloth(cols, rows, ks=(40.0, 30.0, 20.0), size=4.0)
    edge = (sp["type"] == 0) & (sp["p1"] < cols) & (sp["p2"] < cols)
    assert edge.sum() == cols - 1
    sp["rest_length"][edge] *= np.float32(0.75)
    sp["ks"][edge] = ks_edge
    return ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0, cols - 1], np.int32), cg_max_iter=5), X


@pytest.mark.parametrize("ks_edge", [40.0, 80.0])
@pytest.mark.parametrize("cols,rows", [(33, 17), (9, 9), (128, 20), (129, 12)])
def test_rest_lengths_by_class(cols, rows, ks_edge):
    d, X = cloth(cols, rows, ks_edge)
    V = np.random.default_rng(3).normal(0, 0.2, X.shape).astype(np.float32)
    uniform, _ = cloth(cols, rows, 40.0)
    with ClothSolver(d, use_graph=False) as s:
        s.set_spring_params(ks=uniform.springs["ks"])
        s.set_state(X, V)
        s.step(DT, 2)
        a = s.get_state()
        assert ("k_assemble_kinds" in s.profile(DT, 1)) == (cols <= 128)
        # and back: two Ks in a kind leave the kernel again
        s.set_spring_params(ks=d.springs["ks"])
        s.set_state(X, V, np.zeros_like(X))
        s.step(DT, 2)
        b = s.get_state()
        assert ("k_assemble_kinds" in s.profile(DT, 1)) == (cols <= 128 and ks_edge == 40.0)
    for got, desc in ((a, uniform), (b, d)):
        for x, y, z in zip(got, run([desc], X, V, 1)[0], run([desc], X, V, 0)[0]):
            assert np.array_equal(x, y) and np.array_equal(x, z)
