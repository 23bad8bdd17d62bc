"""Handles in which small cloths join larger ones in one k_cg_persist launch, and those short of the
rule, against the WHILE-loop CG (persist 0): the same bits, for the step and for a gradient."""
import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, ClothSolver, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


@pytest.mark.parametrize("shapes,join", [
    ([(150, 150), (9, 9)], True), ([(150, 150), (60, 40), (128, 128), (5, 6)], True),
    ([(130, 127)] + [(20 + k, 41) for k in range(63)], True),
    ([(130, 127)] + [(20 + k % 50, 41) for k in range(64)], False),   # more cloths than the rule takes
    ([(500, 500)] + [(9, 9)] * 60, False),                            # cut unevenly
    ([(100, 100), (9, 9)], None),                                     # all small (k_sim)
    ([(16 + 3 * k, 14 + 3 * (k * 7 % 36)) for k in range(36)], True),  # all small, many sizes
    ([(91, 90)] * 24, False),                                         # all small, one size
    ([(64, 64)], None), ([(64, 64), (40, 40), (30, 20)], None),       # one launch for the solves alone
])
def test_routes_and_bits(shapes, join):
    descs, X = [], []
    for k, (cols, rows) in enumerate(shapes):
        x, sp = grid_cloth(cols, rows, jitter=1e-2, seed=k, ks=(40.0, 40.0, 40.0))
        descs.append(ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0], np.int32), cg_max_iter=3 + k % 4,
                               cg_tol=1e-6))
        X.append(x)
    X = np.concatenate(X)
    V = np.random.default_rng(1).normal(0, 0.1, X.shape).astype(np.float32)
    out = []
    for persist in (1, 0):
        with ClothSolver(descs) as s:
            s.set_launch_config(persist=persist)
            if persist and join is not None:
                prof = s.profile(DT, 1)
                assert ("k_resident" not in prof or prof["k_resident"]["launches"] == 0) == join
            s.set_state(X, V)
            s.step(DT, 3)
            it, _, flags = s.stats()
            state = s.get_state()
            s.set_state(X, V)
            s.tape_forward(DT, 2)
            out.append((*state, it, flags, *s.tape_backward(X).values()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("shapes", [[(21, 21)], [(21, 21), (40, 40), (70, 61)], [(64, 64)] * 8, [(48, 48)] * 48])
def test_single_steps(shapes):
    """Steps one by one (several k_sim launches go as a graph then, rebuilt for another dt) against
    the same steps in one call, and k_sim's plans around the clusters that run at once."""
    descs, X = [], []
    for k, (cols, rows) in enumerate(shapes):
        x, sp = grid_cloth(cols, rows, jitter=1e-2, seed=k)
        descs.append(ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0], np.int32), cg_max_iter=5, cg_tol=1e-5))
        X.append(x)
    X = np.concatenate(X)
    out = []
    for one in (True, False):
        with ClothSolver(descs) as s:
            s.set_state(X, np.zeros_like(X))
            for dt in (DT, 0.5 * DT, DT):
                for n in ([1] * 3 if one else [3]):
                    s.step(dt, n)
            out.append((*s.get_state(), s.stats()[0]))
            n0 = s.launch_count()
            s.step(DT, 1)
            assert s.launch_count() > n0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
