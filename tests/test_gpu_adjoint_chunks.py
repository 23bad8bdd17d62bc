"""The reverse pass's vertex and spring kernels in chunks of 128 vertices: a cloth's gradients do
not depend on what shares its handle, so each cloth of a handle (chunks and blocks that end in
between, incidence records and stencils, rows with more records than a chunk's copies hold) gives the
bits that it gives alone."""
import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, ClothSolver, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def cloth(cols, rows, k):
    X, sp = grid_cloth(cols, rows, jitter=1e-2, seed=k)
    return ClothDesc(n_vertices=cols * rows, springs=sp, pinned=np.array([0, cols - 1], np.int32), cg_max_iter=20), X


def star(n, k):
    """A vertex joined to all others, so the chunk's records exceed its copies."""
    rng = np.random.default_rng(k)
    X = rng.normal(0, 1, (n, 3)).astype(np.float32) + np.float32([0, 5, 0])
    _, sp = grid_cloth(3, 3)
    ends = [(i, i + 1) for i in range(n - 1)] + [(0, i) for i in range(2, n)] + [(1, i) for i in range(3, n)]
    out = np.zeros(len(ends), sp.dtype)
    for s, (p, q) in zip(out, ends):
        s["p1"], s["p2"], s["rest_length"], s["ks"], s["kd"] = p, q, np.linalg.norm(X[p] - X[q]) * 0.98, 0.5, -0.1
    return ClothDesc(n_vertices=n, springs=out, pinned=np.array([0], np.int32), cg_max_iter=20), X


def grads(parts, scale, per_spring):
    descs, X = [p[0] for p in parts], np.concatenate([p[1] for p in parts])
    with ClothSolver(descs) as s:
        if per_spring:
            s.set_spring_params(ks=np.concatenate([d.springs["ks"] * scale[:len(d.springs)] for d in descs]))
        s.set_state(X, np.zeros_like(X))
        s.tape_forward(DT, 3)
        return s.tape_backward(np.sin(100 * X).astype(np.float32))


@pytest.mark.parametrize("per_spring", [False, True])
def test_each_cloth_as_alone(per_spring):
    parts = [cloth(3, 3, 0), cloth(16, 8, 1), cloth(43, 3, 2), star(700, 3), cloth(40, 31, 4), cloth(90, 61, 5), star(150, 6)]
    scale = np.random.default_rng(7).uniform(0.5, 2, 100000).astype(np.float32)
    together = grads(parts, scale, per_spring)
    v = s = 0
    for p in parts:
        alone = grads([p], scale, per_spring)
        nv, ns = p[0].n_vertices, len(p[0].springs)
        for name, g in alone.items():
            o, n = (v, nv) if len(g) == nv else (s, ns)
            assert np.array_equal(g, together[name][o:o + n]), name
        v += nv
        s += ns
