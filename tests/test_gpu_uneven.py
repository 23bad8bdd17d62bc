"""Handles of one large cloth or system beside many small ones in the solves of one launch: the bits of
the loop of separate launches, and not a time that the one CTA left for the large one makes (the limit
is three times the loop's; the CTAs of a plan without regard to it took ten times and more)."""
import time

import numpy as np
import pytest

from opencloth_gb300 import JAC_COUPLED, ClothDesc, ClothSolver, grid_cloth
from opencloth_gb300.fem import BsrSolver, fem_system

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def best(step, wait, n=5):
    ts = []
    for _ in range(n):
        wait()
        t = time.perf_counter()
        step()
        wait()
        ts.append(time.perf_counter() - t)
    return min(ts)


def cloths(shapes, **kw):
    grids = [grid_cloth(c, r, ks=(50.75, 50.75, 50.95), jitter=1e-3, seed=k) for k, (c, r) in enumerate(shapes)]
    return ([ClothDesc(n_vertices=len(X), springs=sp, pinned=np.array([0, c - 1], np.int32), cg_tol=1e-5, **kw)
             for (X, sp), (c, _) in zip(grids, shapes)], np.concatenate([g[0] for g in grids]))


def check_cloths(shapes, **kw):
    descs, X = cloths(shapes, **kw)
    V = np.random.default_rng(5).normal(0, 0.05, X.shape).astype(np.float32)
    out, t = [], []
    for persist in (1, 0):
        with ClothSolver(descs) as s:
            s.set_launch_config(persist=persist)
            s.set_state(X, V)
            s.step(DT, 2)
            it, _, fl = s.stats()
            out.append((*s.get_state(), it, fl))
            t.append(best(lambda: s.step(DT, 3), s.synchronize))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    assert t[0] < 3 * t[1], t


@pytest.mark.parametrize("large,count", [(700, 151), (700, 120), (300, 150), (400, 60)])
def test_reference(large, count):
    check_cloths([(large, large)] + [(130, 130)] * count, cg_max_iter=200)


@pytest.mark.parametrize("large,count", [(500, 150), (500, 60), (200, 151), (200, 120)])
def test_coupled(large, count):
    check_cloths([(large, large)] + [(30, 30)] * count, cg_max_iter=10, jacobian_mode=JAC_COUPLED)


@pytest.mark.parametrize("count", [151, 120])
def test_fem(count):
    """(Without a graph the loop is driven from the host: the time is held against the large system's alone.)"""
    large, small = fem_system(64, 24, 24), fem_system(16, 6, 6)

    def solver(systems, **kw):
        s = BsrSolver(systems, executor=1, **kw)
        s.set_system(*(np.concatenate([g[k] for g in systems]) for k in ("blocks", "b", "V")))
        s.solve()
        return s

    with solver([large] + [small] * count) as s, solver([large] + [small] * count, use_graph=False) as t, solver([large]) as u:
        assert all(np.array_equal(a, b) for a, b in zip(s.solution(), t.solution()))
        ts, tu = (best(x.solve, x.synchronize) for x in (s, u))
    assert ts < 6 * tu, (ts, tu)
