"""The COUPLED CG in one cooperative launch (k_cpl_persist) against the WHILE loop of its two
kernels (persist 0): the same vertex arithmetic in the same order, scalars that differ only beyond
their floats' digits, so the same bits, flags and iteration counts.  Vertex counts around a CTA's
smallest piece and threads, cloths beyond what shared memory holds, several cloths that end at
different iterations, other cloths beside them, and more cloths than SMs (the loop)."""
import numpy as np
import pytest

from opencloth_gb300 import JAC_COUPLED, PASS_PROVOT, ClothDesc, ClothSolver, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def cloth(cols, rows, seed, pinned=(0,), mode=JAC_COUPLED, **kw):
    X, sp = grid_cloth(cols, rows, jitter=1e-2, seed=seed)
    kw = {"cg_max_iter": 7, "cg_tol": 1e-6, **kw}
    d = ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array(sorted(set(p % (cols * rows) for p in pinned)), np.int32),
                  jacobian_mode=mode, **kw)
    return d, X


def check(parts, steps=3, **kw):
    X = np.concatenate([p[1] for p in parts])
    V = np.random.default_rng(4).normal(0, 0.05, X.shape).astype(np.float32)
    out = []
    for persist in (1, 0):
        with ClothSolver([p[0] for p in parts], **kw) as s:
            s.set_launch_config(persist=persist)
            s.set_state(X, V)
            s.step(DT, 1)
            s.step(DT, steps - 1)
            it, rr, fl = s.stats()
            out.append((*s.get_state(), it, fl, rr))
    for a, b in zip(out[0][:5], out[1][:5]):
        assert np.array_equal(a, b, equal_nan=True)
    # r.z itself: float pairs (about 48 bits) against FP64 above a warp.
    np.testing.assert_allclose(out[0][5], out[1][5], rtol=2.0**-40, atol=0)
    return out[0]


@pytest.mark.parametrize("cols,rows", [(3, 3), (15, 17), (16, 16), (16, 17), (32, 31), (33, 31), (65, 63), (200, 199)])
def test_sizes(cols, rows):
    check([cloth(cols, rows, cols, pinned=(0, cols - 1))])


def test_beyond_shared_memory():
    """About 3,500 vertices a CTA, more than its shared memory holds, and a second odd cloth."""
    check([cloth(700, 699, 3, cg_max_iter=4), cloth(211, 203, 4)], steps=2)


def test_stop_rules_and_a_wholly_pinned_cloth():
    parts = [cloth(40, 41, 1, cg_max_iter=200, cg_tol=1e-3), cloth(61, 33, 2, cg_max_iter=1), cloth(30, 30, 3, cg_max_iter=0),
             cloth(10, 9, 4, pinned=range(90)), cloth(50, 20, 5, cg_max_iter=60, cg_tol=1e-5, passes=PASS_PROVOT)]
    it = check(parts)[3]
    assert len(set(it.tolist())) > 2


def test_beside_resident_and_streamed_cloths():
    check([cloth(45, 44, 1), cloth(20, 21, 2, mode=0), cloth(31, 30, 3)])
    check([cloth(45, 44, 1), cloth(200, 180, 2, mode=0), cloth(20, 21, 3, mode=0)])
    check([cloth(45, 44, 1), cloth(20, 21, 2, mode=0)], executor="streamed")


@pytest.mark.parametrize("count", [150, 160])
def test_many_cloths(count):
    check([cloth(5 + k % 9, 6 + k % 7, k, cg_max_iter=2 + k % 6) for k in range(count)], steps=2)


def test_one_launch_for_the_loop():
    d, X = cloth(90, 80, 1)
    with ClothSolver(d) as s:
        s.set_state(X, np.zeros_like(X))
        s.step(DT, 1)
        n = s.launch_count()
        s.step(DT, 5)
        assert s.launch_count() - n == 10  # assembly and CG


def test_a_wait_that_runs_out_is_reported():
    from opencloth_gb300 import OcError
    from opencloth_gb300 import _native as N

    d, X = cloth(70, 70, 2)
    with ClothSolver(d) as s, ClothSolver(d) as t:
        for h in (s, t):
            h.set_state(X, np.zeros_like(X))
            h.step(DT, 1)
        before = s.get_state()
        assert N.load().oc_test_barrier_timeout(s._h, 1, 2000) == 0
        s.step(DT, 1)
        with pytest.raises(OcError) as e:
            s.synchronize()
        assert e.value.status == 8
        assert all(np.array_equal(a, b) for a, b in zip(before[:2], s.get_state()[:2]))  # no update applied
        assert N.load().oc_test_barrier_timeout(s._h, -1, 0) == 0
        s.set_state(*t.get_state())
        s.step(DT, 3)
        t.step(DT, 3)
        assert all(np.array_equal(a, b) for a, b in zip(s.get_state(), t.get_state()))
