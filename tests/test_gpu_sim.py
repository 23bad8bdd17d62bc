"""Whole steps in one launch (k_sim, oc_sim.cu): the bits, iteration counts and flags of the same
cloths stepped by the separate launches (executor "streamed": assembly and persistent CG), at the
edges of its launch shapes (256, 512 and 1024 vertices a CTA, one CTA to sixteen), for grids with
and without exact spacing, general meshes, the passes, and every way a CG ends."""
import numpy as np
import pytest

from opencloth_gb300 import (PASS_ELLIPSOID, PASS_PROVOT, SPRING_DTYPE, ClothDesc, ClothSolver, grid_cloth,
                             reference_ellipsoid)

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def same_bits(a, b) -> bool:
    return np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))


def grid(cols, rows, seed, jitter=1e-2, ks=(50.75, 50.75, 50.95), **kw):
    rng = np.random.default_rng(seed)
    X, sp = grid_cloth(cols, rows, ks=ks, kd=(-0.25, -0.25, -0.25), jitter=jitter, seed=seed)
    V = rng.normal(0.0, 0.05, X.shape).astype(np.float32)
    pins = np.array([0, cols - 1], np.int32)
    V[pins] = 0.0
    return ClothDesc(n_vertices=len(X), springs=sp, pinned=pins, **{"cg_max_iter": 200, "cg_tol": 1e-5, **kw}), X, V


def mesh(n, seed, springs_per_vertex=4):
    """A general cloth: random springs (so neighbours lie in any CTA), masses, pins, an external
    force, and fewer springs than vertices when springs_per_vertex is below one."""
    rng = np.random.default_rng(seed)
    X = rng.uniform(0.5, 4.0, (n, 3)).astype(np.float32)
    m = max(1, int(n * springs_per_vertex))
    a = rng.integers(0, n, m)
    b = (a + 1 + rng.integers(0, n - 1, m)) % n
    sp = np.zeros(m, SPRING_DTYPE)
    sp["p1"], sp["p2"] = a, b
    sp["rest_length"] = np.linalg.norm(X[a] - X[b], axis=1) * rng.uniform(0.9, 1.1, m)
    sp["ks"], sp["kd"] = rng.uniform(5, 50, m), -0.25
    V = rng.normal(0, 0.05, X.shape).astype(np.float32)
    pins = np.unique(rng.integers(0, n, max(1, n // 50))).astype(np.int32)
    return ClothDesc(n_vertices=n, springs=sp, pinned=pins, mass=rng.uniform(0.5, 2, n).astype(np.float32),
                     ext_force=rng.normal(0, 0.1, (n, 3)).astype(np.float32), cg_max_iter=200, cg_tol=1e-5), X, V


def stepped(parts, calls, executor):
    descs = [p[0] for p in parts]
    X, V = np.concatenate([p[1] for p in parts]), np.concatenate([p[2] for p in parts])
    with ClothSolver(descs, executor=executor) as s:
        s.set_state(X, V)
        for n in calls:
            s.step(DT, n)
        return s.get_state(), s.stats()


def check(parts, calls=(3, 1)):
    a, sa = stepped(parts, calls, "auto")
    b, sb = stepped(parts, (sum(calls),), "streamed")
    for x, y in zip(a, b):
        assert same_bits(x, y)
    assert np.array_equal(sa[0], sb[0]) and np.array_equal(sa[2], sb[2])
    return sa


SIZES = [(3, 3), (4, 5), (16, 16), (257, 3), (3, 171), (21, 21), (64, 64), (4097, 3), (91, 45), (128, 64), (121, 71),
         (128, 128), (127, 129)]


@pytest.mark.parametrize("cols,rows", SIZES, ids=lambda v: str(v))
def test_grid_sizes(cols, rows):
    check([grid(cols, rows, cols + rows)])


@pytest.mark.parametrize("n", [2, 31, 256, 257, 1000, 4097, 9001, 16384])
def test_general_meshes(n):
    check([mesh(n, n)])


def test_fewer_springs_than_vertices():
    check([mesh(700, 5, 0.4)])


@pytest.mark.parametrize("cols,rows,jitter", [(21, 21, 0.0), (40, 33, 1e-2), (101, 90, 1e-2)])
def test_passes(cols, rows, jitter):
    E, Einv = reference_ellipsoid()
    d, X, V = grid(cols, rows, 9, jitter, ks=(5.0, 5.0, 5.0), passes=PASS_ELLIPSOID | PASS_PROVOT, ellipsoid=E,
                   ellipsoid_inv=Einv)
    X = X.copy()
    X[:, 1] -= 2.0
    check([(d, X, V)], (4, 3))


def test_mesh_with_provot():
    d, X, V = mesh(1500, 8)
    d.passes = PASS_PROVOT
    check([(d, X, V)], (2, 2))


def test_several_cloths_of_every_shape():
    check([grid(17, 23, 1), grid(90, 60, 2), grid(128, 100, 3), mesh(300, 4), grid(64, 64, 5), mesh(5000, 6)])


def test_ends_of_the_cg():
    """Converged, the iteration cap, no iterations, an indefinite system, a cloth at rest."""
    parts = [grid(30, 20, 1), grid(30, 20, 2, cg_max_iter=1, cg_tol=1e-9), grid(30, 20, 3, cg_max_iter=0),
             grid(30, 20, 4, ks=(5e5, 5e5, 5e5), cg_max_iter=50, cg_tol=1e-9)]
    it, _, fl = check(parts, (1, 1))
    assert it[0] > 1 and fl[0] == 0 and it[1] == 1 and fl[1] & 1 and it[2] == 0
    rest = grid(20, 20, 5, 0.0, gravity=(0.0, 0.0, 0.0))
    it, _, fl = check([(rest[0], rest[1], np.zeros_like(rest[1]))], (2,))


def test_long_call_equals_many_short_ones():
    parts = [grid(21, 21, 3), grid(50, 40, 4)]
    a, _ = stepped(parts, (520,), "auto")  # more steps than one launch takes
    b, _ = stepped(parts, (1,) * 8 + (512,), "auto")
    for x, y in zip(a, b):
        assert same_bits(x, y)
