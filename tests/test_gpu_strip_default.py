"""The handles that take the strip sweep by themselves (large ones whose grid cloths all suit it)
and those just short of it, against k_assemble_grid: F, A and b are the same bits, delta0 is summed
in another order (float pairs), so the state comes out the same."""
import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, ClothSolver, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


@pytest.mark.parametrize("shapes,strip", [
    ([(420, 419)], 1),                       # 175,980 vertices
    ([(418, 418)], 0),                       # 174,724
    ([(1009, 175)], 1), ([(175, 1009)], 1),  # odd sides
    ([(55, 57)] * 57, 1),                    # resident cloths: k_assemble_finish forms their delta0
    ([(600, 400), (41, 40)], 0),             # a cloth whose lanes would idle
    ([(600, 400), (56, 55)], 1),
])
def test_default_and_bits(shapes, strip):
    descs, X = [], []
    for k, (cols, rows) in enumerate(shapes):
        x, sp = grid_cloth(cols, rows, jitter=1e-2, seed=k)
        descs.append(ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0, cols - 1], np.int32),
                               cg_max_iter=6, cg_tol=1e-6))
        X.append(x)
    X = np.concatenate(X)
    V = np.random.default_rng(1).normal(0, 0.1, X.shape).astype(np.float32)
    out = []
    for other in (None, 1 - strip):
        with ClothSolver(descs) as s:
            assert s.launch_config()["strip"] == strip
            if other is not None:
                s.set_launch_config(strip=other)
            s.set_state(X, V)
            s.step(DT, 2)
            out.append(s.get_state())
    for a, b in zip(*out):
        assert np.array_equal(a, b)
