"""The bytes the profile counts for the solves that keep their state on chip: what a launch has to move,
and not what the loop of separate kernels would."""
import numpy as np
import pytest

from opencloth_gb300 import JAC_COUPLED, ClothDesc, ClothSolver, grid_cloth, grid_spring_count

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def counted(cols, rows, iters, kernel, **kw):
    X, sp = grid_cloth(cols, rows, ks=(50.75, 50.75, 50.95), jitter=1e-2, seed=1)
    V = np.random.default_rng(2).normal(0, 0.05, X.shape).astype(np.float32)
    d = ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0, cols - 1], np.int32), cg_max_iter=iters,
                  cg_tol=1e-9, **kw)
    with ClothSolver(d) as s:
        s.set_state(X, V)
        p = s.profile(DT, 1)[kernel]
        assert p["launches"] == 1 and s.stats()[0][0] == iters
        return p["bytes"]


@pytest.mark.parametrize("cols,rows", [(257, 250), (449, 447), (1025, 700)])
def test_persistent_cg_on_chip(cols, rows):
    """The CG state and X, V in, x, X and V out, 136 bytes a vertex, whatever the iterations."""
    assert [counted(cols, rows, k, "k_cg_persist") for k in (1, 2, 5)] == [136.0 * cols * rows] * 3


def test_persistent_cg_with_slots_in_the_planes():
    cols, rows = 1300, 1200  # 41 slots a CTA of 33 on chip
    b = [counted(cols, rows, k, "k_cg_persist") / (cols * rows) for k in (1, 2, 3)]
    assert b[0] > 136.0 and b[1] > b[0] and abs((b[2] - b[1]) - (b[1] - b[0])) < 13.0
    assert b[2] < 36.0 + 60.0 * 2 + 84.0 * 3 + 76.0  # less than the loop's


@pytest.mark.parametrize("cols,rows", [(60, 70), (513, 500)])
def test_coupled_cg(cols, rows):
    """An iteration: a block (24 bytes) at each end of each spring, z, d, counts and flags of a vertex."""
    n, ns = cols * rows, grid_spring_count(cols, rows)
    b = [counted(cols, rows, k, "k_cpl_persist", jacobian_mode=JAC_COUPLED) for k in (1, 2, 3)]
    assert b[2] - b[1] == b[1] - b[0] == 73.0 * n + 48.0 * ns
    assert b[0] == 185.0 * n + 48.0 * ns
