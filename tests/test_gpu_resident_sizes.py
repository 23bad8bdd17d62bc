"""The resident CG (k_resident) at the edges of its CTAs and clusters against the streamed
executor: the same FP32 arithmetic a vertex, sums that differ beyond their floats' digits, so the
same bits.  Stepped launch by launch, so that small handles too run k_resident."""
import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, ClothSolver, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def parts(shapes, **kw):
    out = []
    for k, (cols, rows) in enumerate(shapes):
        X, sp = grid_cloth(cols, rows, jitter=1e-2, seed=k, ks=(50.0, 50.0, 50.0))
        out.append((ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0], np.int32),
                              **{"cg_max_iter": 9, "cg_tol": 1e-6, **kw}), X))
    return [p[0] for p in out], np.concatenate([p[1] for p in out])


def run(descs, X, executor):
    with ClothSolver(descs, executor=executor, use_graph=False) as s:
        s.set_state(X, np.random.default_rng(2).normal(0, 0.1, X.shape).astype(np.float32))
        s.step(DT, 3)
        it, _, flags = s.stats()
        return (*s.get_state(), it, flags)


@pytest.mark.parametrize("shape", [(3, 3), (31, 33), (32, 32), (25, 41), (64, 32), (3, 683), (111, 83), (127, 129), (128, 128)])
@pytest.mark.parametrize("imax", [0, 1, 9])
def test_sizes(shape, imax):
    descs, X = parts([shape], cg_max_iter=imax)
    for a, b in zip(run(descs, X, "resident"), run(descs, X, "streamed")):
        assert np.array_equal(a, b)


def test_many_clusters_of_every_size():
    descs, X = parts([(64, 16 * c + d) for c in range(1, 17) for d in (0, -1, -7)] * 4)
    for a, b in zip(run(descs, X, "resident"), run(descs, X, "streamed")):
        assert np.array_equal(a, b)
