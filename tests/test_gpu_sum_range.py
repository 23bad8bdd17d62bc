"""Dot products whose terms are finite floats but whose total lies beyond the largest one: the solves
in one launch (k_cg_persist, k_cpl_persist, k_bsr_persist, k_bsr_resident), whose sums travel as
float pairs, go on like the loops that add up in FP64.  Each system is scaled up step by step, through
the range where only the total is out of float's, until the loop's own sums of a warp are: state,
iterations and flags are compared at every step where the loop ends well."""
import numpy as np
import pytest

from opencloth_gb300 import FLAG_BREAKDOWN, FLAG_NON_FINITE, JAC_COUPLED, ClothDesc, ClothSolver, grid_cloth
from opencloth_gb300.fem import BsrSolver
from test_gpu_fem_resident import system

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def stepped(descs, X, V, persist, **kw):
    with ClothSolver(descs, **kw) as s:
        s.set_launch_config(persist=persist)
        s.set_state(X, V)
        s.step(DT, 1)
        it, _, fl = s.stats()
        return (*s.get_state(), it, fl)


def scan(make, steps, **kw):
    flags = []
    for k in steps:
        descs, X, V = make(k)
        a, b = (stepped(descs, X, V, p, **kw) for p in (1, 0))
        flags.append(int(b[4].max()) & (FLAG_NON_FINITE | FLAG_BREAKDOWN))
        assert flags[-1] or all(np.array_equal(x, y) for x, y in zip(a, b)), k
    assert flags[0] == 0 and flags[-1] != 0
    return flags


@pytest.mark.parametrize("shapes", [[(40, 50)], [(257, 250)], [(449, 447)], [(1025, 700)], [(30 + k % 9, 40) for k in range(200)]],
                         ids=["a cluster", "clusters", "registers", "pairs", "pieces"])
def test_reference(shapes):
    """Gravity times 2^k on cloths at rest: r.r and d.(A d) grow as 2^2k."""
    grids = [grid_cloth(c, r, ks=(50.75, 50.75, 50.95)) for c, r in shapes]
    X = np.concatenate([g[0] for g in grids])

    def make(k):
        return ([ClothDesc(n_vertices=c * r, springs=g[1], pinned=np.array([0, c - 1], np.int32), cg_max_iter=30,
                           cg_tol=1e-5, gravity=(0.0, -9.81e-3 * 2.0**k, 0.0)) for g, (c, r) in zip(grids, shapes)],
                X, np.zeros_like(X))

    scan(make, range(54, 76), executor="streamed")


@pytest.mark.parametrize("cols,rows", [(60, 70), (257, 250)])
def test_coupled(cols, rows):
    """Gravity times 2^k on a cloth at rest: r.z grows as 2^2k."""
    X, sp = grid_cloth(cols, rows)

    def make(k):
        return ([ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0, cols - 1], np.int32), cg_max_iter=6,
                           cg_tol=1e-9, gravity=(0.0, -9.81e-3 * 2.0**k, 0.0), jacobian_mode=JAC_COUPLED)], X, np.zeros_like(X))

    scan(make, range(50, 76))


@pytest.mark.parametrize("n,executor", [(2000, 1), (9000, 1), (200, 2)])
def test_fem(n, executor):
    """The matrix and the right-hand side times 2^(j/4): p.q grows as its cube."""
    g = system(n, n, 9, i_max=4)
    arrays = [g[k] for k in ("blocks", "b", "V")]
    finite = []
    for j in range(100, 190):
        f = np.float32(2.0 ** (j / 4))
        out = []
        for kw in (dict(executor=executor), dict(executor=1, use_graph=False)):
            with BsrSolver([g], **kw) as s:
                s.set_system(arrays[0] * f, arrays[1] * f, arrays[2])
                s.solve()
                out.append(s.solution())
        finite.append(bool(np.isfinite(out[1][0]).all()))
        assert not finite[-1] or all(np.array_equal(a, b) for a, b in zip(*out)), j
    assert finite[0] and not finite[-1]
