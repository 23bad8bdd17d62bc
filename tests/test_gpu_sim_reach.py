"""Grid cloths whose springs go further than the reference's (two rows and two columns at once, a
knight's move) in k_sim, whose window has to reach as far as the stencil: the bits of the streamed
executor, on one CTA and on several, with and without Provot's pass."""
import numpy as np
import pytest

from opencloth_gb300 import PASS_PROVOT, SPRING_DTYPE, ClothDesc, describe, grid_cloth
from test_gpu_sim import check

pytestmark = pytest.mark.gpu

DIAGONAL = [(2, 2), (2, -2)]
KNIGHT = [(2, 1), (2, -1), (1, 2), (1, -2)]


def cloth(cols, rows, extra, jitter, passes):
    X, sp = grid_cloth(cols, rows, ks=(5.0, 4.0, 3.0), kd=(-0.25, -0.25, -0.25), jitter=jitter, seed=cols)
    more = []
    for dr, dc in extra:
        r, c = np.meshgrid(np.arange(rows - dr), np.arange(max(0, -dc), cols - max(0, dc)), indexing="ij")
        t = np.zeros(r.size, SPRING_DTYPE)
        t["p1"], t["p2"] = (r * cols + c).ravel(), ((r + dr) * cols + c + dc).ravel()
        t["ks"], t["kd"] = 2.0, -0.2
        if jitter:
            t["rest_length"] = np.linalg.norm(X[t["p1"]] - X[t["p2"]], axis=1)
        else:
            t["rest_length"] = np.hypot(dr, dc) * 4.0 / (cols - 1)
        more.append(t)
    d = ClothDesc(n_vertices=cols * rows, springs=np.concatenate([sp, *more]), cg_max_iter=200, cg_tol=1e-5,
                  pinned=np.array([0, cols - 1], np.int32), passes=passes, provot_ratio=1.0)
    V = np.random.default_rng(rows).normal(0.0, 0.3, X.shape).astype(np.float32)
    V[[0, cols - 1]] = 0.0
    return d, X, V


@pytest.mark.parametrize("passes", [0, PASS_PROVOT])
@pytest.mark.parametrize("extra", [DIAGONAL, KNIGHT, KNIGHT + DIAGONAL], ids=["diagonal", "knight", "both"])
@pytest.mark.parametrize("cols,rows,jitter", [(21, 21, 0.0), (30, 30, 1e-2), (100, 75, 0.0), (9, 400, 1e-2)])
def test_springs_that_reach_further(cols, rows, jitter, extra, passes):
    d, X, V = cloth(cols, rows, extra, jitter, passes)
    assert describe([d]) == [(cols, rows)]
    check([(d, X, V)], (3, 1))
