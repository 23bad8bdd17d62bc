"""The streamed CG of handles whose state k_cg_persist cannot hold on chip (k_cg_arrive): the bits,
iterations and flags of the two-kernel loop, on both sides of the rule that chooses between the two;
its gradients; and its bounded waits."""
import os

import numpy as np
import pytest

from opencloth_gb300 import ClothSolver, OcError
from opencloth_gb300 import _native as N
from test_gpu_persist import cloth, run, same_bits

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0

HANDLES = {
    "tiny": [(8, 8)] * 4000,  # 27 slots and 27 pieces a CTA
    "ragged": [(8 + k % 17, 8 + k % 13) for k in range(3600)],
    "large": [(1600, 1500)],
    "several large": [(900, 800), (700, 900), (1100, 1000), (60, 50)],
    "many": [(130, 128 + k % 5) for k in range(112)],
    "many on chip": [(130, 128 + k % 5) for k in range(84)],
    "uneven": [(1100, 1000)] + [(130, 130)] * 100,
}


def parts(name):
    ps = [cloth(c, r, k, ks=(50.75, 50.75, 50.95) if k % 3 else (300.0, 200.0, 400.0)) for k, (c, r) in enumerate(HANDLES[name])]
    return [p[0] for p in ps], np.concatenate([p[1] for p in ps]), np.concatenate([p[2] for p in ps])


@pytest.mark.parametrize("name", HANDLES)
def test_same_bits(name):
    descs, X, V = parts(name)
    kw = dict(executor="streamed")
    a, sa = run(descs, X, V, 2, True, **kw)
    b, sb = run(descs, X, V, 2, False, **kw)
    assert all(same_bits(x, y) for x, y in zip(a, b))
    assert np.array_equal(sa[0], sb[0]) and np.array_equal(sa[2], sb[2]) and sa[0].max() > 1
    with ClothSolver(descs, **kw) as s:
        s.set_state(X, V)
        s.step(DT, 1)
        n = s.launch_count()
        s.step(DT, 2)
        assert s.launch_count() - n == 4  # the assembly and the CG
        names = s.profile(DT, 1)
        assert ("k_cg_persist" in names) == (name == "many on chip") and ("k_cg_arrive" in names) != ("k_cg_persist" in names)


def test_gradients():
    descs, X, V = parts("tiny")
    g = np.random.default_rng(1).normal(0, 1, X.shape).astype(np.float32)
    out = []
    for persist in ("1", "0"):
        os.environ["OC_PERSIST"] = persist
        try:
            with ClothSolver(descs, executor="streamed") as s:
                s.set_state(X, V, np.zeros_like(X))
                s.tape_forward(DT, 3)
                out.append(s.tape_backward(g))
        finally:
            os.environ.pop("OC_PERSIST")
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


def test_a_wait_that_runs_out_is_reported():
    descs, X, V = parts("tiny")
    # one cloth of several blocks among them, whose blocks wait for one another
    d, X1, V1 = cloth(200, 150, 9)
    descs, X, V = [d] + descs, np.concatenate([X1, X]), np.concatenate([V1, V])
    lib = N.load()
    with ClothSolver(descs, executor="streamed") as s, ClothSolver(descs, executor="streamed") as t:
        for h in (s, t):
            h.set_state(X, V)
            h.step(DT, 1)
        assert "k_cg_arrive" in t.profile(DT, 1)
        t.set_state(*s.get_state())
        before = s.get_state()
        assert lib.oc_test_barrier_timeout(s._h, 1, 2000) == 0
        s.step(DT, 1)
        with pytest.raises(OcError) as e:
            s.synchronize()
        assert e.value.status == 8
        n = d.n_vertices
        assert all(same_bits(a[:n], b[:n]) for a, b in zip(before[:2], s.get_state()[:2]))
        assert lib.oc_test_barrier_timeout(s._h, -1, 0) == 0
        s.set_state(*before)
        s.step(DT, 2)
        t.step(DT, 2)
        assert all(same_bits(a, b) for a, b in zip(s.get_state(), t.get_state()))


@pytest.mark.parametrize("large,small", [([(1250, 1240)], 35), ([(1500, 1400)], 20), ([(500, 400)] * 6, 10), ([(500, 400)] * 5, 100)])
def test_beside_small_cloths(large, small):
    """Cloths for both kernels with small ones that join them or run resident beside them."""
    ps = [cloth(c, r, k) for k, (c, r) in enumerate(large + [(20 + 7 * k % 40, 21 + 5 * k % 37) for k in range(small)])]
    descs, X, V = [p[0] for p in ps], np.concatenate([p[1] for p in ps]), np.concatenate([p[2] for p in ps])
    a, sa = run(descs, X, V, 3, True)
    b, sb = run(descs, X, V, 3, False)
    assert all(same_bits(x, y) for x, y in zip(a, b))
    assert np.array_equal(sa[0], sb[0]) and np.array_equal(sa[2], sb[2])
