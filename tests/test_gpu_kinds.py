"""k_assemble_kinds (grid cloths of up to 128 columns in the reference's spring order, from windows
of the states in shared memory) against k_assemble over the incidence records (OC_STENCIL=0): the
same forces added in the same order, so the same bits."""
import os

import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, ClothSolver, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def run(descs, X, V, stencil, **kw):
    os.environ["OC_STENCIL"] = str(stencil)
    try:
        with ClothSolver(descs, use_graph=False, **kw) as s:  # (launch by launch: small handles too)
            s.set_state(X, V)
            s.step(DT, 2)
            out = s.get_state()
            name = "k_assemble_kinds" in s.profile(DT, 1)
    finally:
        os.environ.pop("OC_STENCIL")
    return out, name


def cloths(shapes, jitter, ext=False):
    descs, Xs = [], []
    for k, (cols, rows) in enumerate(shapes):
        X, sp = grid_cloth(cols, rows, jitter=jitter, seed=k, ks=(40.0, 30.0, 20.0))
        rng = np.random.default_rng(k)
        f = rng.normal(0, 0.01, X.shape).astype(np.float32) if ext else None
        descs.append(ClothDesc(n_vertices=cols * rows, springs=sp, ext_force=f,
                               pinned=np.array(sorted({0, cols - 1, (cols * rows) // 2}), np.int32), cg_max_iter=5))
        Xs.append(X)
    X = np.concatenate(Xs)
    return descs, X, np.random.default_rng(9).normal(0, 0.2, X.shape).astype(np.float32)


@pytest.mark.parametrize("shapes", [
    [(3, 3)], [(4, 5)], [(5, 4)], [(8, 64)], [(3, 900)],      # spring i's ends beyond the window
    [(16, 32), (16, 33)], [(127, 40)], [(128, 128)], [(128, 131)], [(64, 500)],
    [(9 + 5 * k % 120, 7 + 11 * k % 90) for k in range(40)],
])
@pytest.mark.parametrize("jitter", [0.0, 1e-2])
def test_same_bits(shapes, jitter):
    descs, X, V = cloths(shapes, jitter, ext=len(shapes) > 1)
    (a, kinds), (b, other) = run(descs, X, V, 1), run(descs, X, V, 0)
    assert kinds and not other
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_springs_out_of_range_and_wider_cloths():
    """A zero-length spring (the general force), and a cloth too wide for the window."""
    descs, X, V = cloths([(20, 20)], 0.0)
    X = X.copy()
    X[45] = X[44]
    X[300] = X[280] + np.float32(1e-25)
    for x, y in zip(run(descs, X, V, 1)[0], run(descs, X, V, 0)[0]):
        assert np.array_equal(x, y, equal_nan=True)
    descs, X, V = cloths([(129, 20), (30, 30)], 1e-2)
    (a, kinds), (b, _) = run(descs, X, V, 1), run(descs, X, V, 0)
    assert not kinds
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_new_spring_parameters():
    """Ks / Kd scaled per spring type keep the kernel, values that differ among a kind's slots or
    springs leave it; each state steps like a handle created with those parameters."""
    descs, X, V = cloths([(4, 5), (40, 30)], 0.0)
    sp = [d.springs for d in descs]
    ks = np.concatenate([s["ks"] for s in sp])
    rng = np.random.default_rng(5)
    rest = np.concatenate([s["rest_length"] for s in sp])
    by_rest = ks * np.where(rest > np.median(rest), 2, 1).astype(np.float32)
    for new, kinds in ((ks * np.float32(1.5), True), (by_rest, None), (ks * rng.uniform(0.5, 2, len(ks)).astype(np.float32), False),
                       (ks, True)):
        with ClothSolver(descs, use_graph=False) as s:
            s.set_spring_params(ks=by_rest)
            s.set_spring_params(ks=new)
            s.set_state(X, V)
            s.step(DT, 2)
            a = s.get_state()
            assert kinds is None or ("k_assemble_kinds" in s.profile(DT, 1)) == kinds
        fresh, o = [], 0
        for d in descs:
            t = d.springs.copy()
            t["ks"] = new[o:o + len(t)]
            o += len(t)
            fresh.append(ClothDesc(n_vertices=d.n_vertices, springs=t, pinned=d.pinned, cg_max_iter=5))
        for x, y in zip(a, run(fresh, X, V, 0)[0]):
            assert np.array_equal(x, y)
