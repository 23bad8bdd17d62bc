"""The bounded waits between CTAs: a CTA that sends no sums makes the others' waits run out after a
short limit of polls, the error is reported once, and the handle then steps on with the bits of one
that never saw it."""
import numpy as np
import pytest

from opencloth_gb300 import PASS_PROVOT, ClothSolver, OcError
from opencloth_gb300 import _native as N
from opencloth_gb300.fem import BsrSolver
from test_gpu_fem_resident import system
from test_gpu_sim import grid, same_bits

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def check(parts, steps, block, polls, **kw):
    X, V = np.concatenate([p[1] for p in parts]), np.concatenate([p[2] for p in parts])
    descs = [p[0] for p in parts]
    lib = N.load()
    with ClothSolver(descs, **kw) as s, ClothSolver(descs, **kw) as t:
        for h in (s, t):
            h.set_state(X, V)
            h.step(DT, 2)
        before = t.get_state()
        assert lib.oc_test_barrier_timeout(s._h, block, polls) == 0
        s.step(DT, steps)
        with pytest.raises(OcError) as e:
            s.synchronize()
        assert e.value.status == 8
        after = s.get_state()  # (reported once)
        n = parts[0][0].n_vertices  # the cloth of block 0 and 1: no sums, so no update
        assert all(same_bits(a[:n], b[:n]) for a, b in zip(before[:2], after[:2]))
        assert lib.oc_test_barrier_timeout(s._h, -1, 0) == 0
        s.set_state(*before)
        for n in (1, 3):
            s.step(DT, n)
            t.step(DT, n)
        for a, b in zip(s.get_state(), t.get_state()):
            assert same_bits(a, b)
        assert np.array_equal(s.stats()[0], t.stats()[0])


@pytest.mark.parametrize("steps", [1, 6])
@pytest.mark.parametrize("polls", [50, 3000])
@pytest.mark.parametrize("block", [0, 1])
@pytest.mark.parametrize("passes", [0, PASS_PROVOT])
@pytest.mark.parametrize("shapes", [[(30, 30)], [(60, 60)] * 3, [(120, 101)] * 5, [(30, 20), (90, 90), (60, 60)]],
                         ids=["two CTAs", "clusters", "of sixteen", "groups"])
def test_whole_steps_in_one_launch(shapes, passes, block, polls, steps):
    """k_sim: CTAs that give up at different exchanges leave their cluster together."""
    check([grid(c, r, k, passes=passes) for k, (c, r) in enumerate(shapes)], steps, block, polls)


@pytest.mark.parametrize("polls", [50, 3000])
@pytest.mark.parametrize("block", [0, 1])
@pytest.mark.parametrize("shapes", [[(30, 30)], [(200, 190)], [(300, 280), (120, 90), (60, 60)],
                                    [(6 + k % 25, 7 + k % 23) for k in range(330)]],
                         ids=["a cluster", "clusters", "several", "pieces"])
def test_persistent_cg(shapes, block, polls):
    check([grid(c, r, k) for k, (c, r) in enumerate(shapes)], 2, block, polls, executor="streamed")


@pytest.mark.parametrize("polls", [50, 3000])
@pytest.mark.parametrize("count", [1, 40])
def test_resident_cg(count, polls):
    """k_resident: a handle without graphs, and more cloths of several CTAs than k_sim takes."""
    parts = [grid(120, 100, 1)] + [grid(70 + k % 3, 60, k) for k in range(count - 1)]
    check(parts, 1, 1, polls, **({"use_graph": False} if count == 1 else {}))


@pytest.mark.parametrize("polls", [50, 3000])
@pytest.mark.parametrize("block", [0, 1])
@pytest.mark.parametrize("sizes", [[3000], [2000, 40, 1500]])
def test_fem_solve(sizes, block, polls):
    systems = [system(n, n, 9, i_max=7) for n in sizes]
    arrays = [np.concatenate([g[k] for g in systems]) for k in ("blocks", "b", "V")]
    lib = N.load()
    with BsrSolver(systems, executor=1) as s:
        s.set_system(*arrays)
        s.solve()
        want = s.solution()
        assert lib.oc_bsr_test_barrier_timeout(s._h, block, polls) == 0
        s.set_system(*arrays)
        s.solve()
        with pytest.raises(OcError) as e:
            s.synchronize()
        assert e.value.status == 8
        s.synchronize()  # (reported once)
        assert lib.oc_bsr_test_barrier_timeout(s._h, -1, 0) == 0
        for _ in range(2):
            s.set_system(*arrays)
            s.solve()
            assert all(np.array_equal(a, b) for a, b in zip(s.solution(), want))
