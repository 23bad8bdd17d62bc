"""The packets' 32-bit tags of the CG launches (k_cg_persist, k_cpl_persist) run on from launch to
launch and wrap after some hours of stepping: handles set to a little before the wrap step across it
with the bits, iterations and flags of fresh ones.  One CTA a cloth, one cluster, several clusters,
pairs of CTAs, several pieces a CTA; from starts that put the tag 0 into every phase of a solve."""
import numpy as np
import pytest

from opencloth_gb300 import JAC_COUPLED, ClothSolver
from opencloth_gb300 import _native as N
from test_gpu_coupled_persist import cloth as coupled
from test_gpu_persist import cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


def stepped(parts, last, replan=False, **kw):
    X = np.concatenate([p[1] for p in parts])
    V = np.random.default_rng(4).normal(0, 0.05, X.shape).astype(np.float32)
    with ClothSolver([p[0] for p in parts], **kw) as s:
        if last is not None:
            s.set_state(X, V)
            s.step(DT, 1)
            assert N.load().oc_test_packet_tags(s._h, last) == 0
        if replan:
            s.set_launch_config(persist=0)
            s.set_launch_config(persist=1)
        s.set_state(X, V, np.zeros_like(X))
        for _ in range(3):
            s.step(DT, 1)
        it, _, fl = s.stats()
        return (*s.get_state(), it, fl)


def check(parts, **kw):
    want = stepped(parts, None, **kw)
    assert want[3].max() > 1
    for before in range(1, 14):
        got = stepped(parts, 2**32 - before, **kw)
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), before
    got = stepped(parts, 2**32 - 3, replan=True, **kw)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("shapes", [
    [(15, 14)], [(50, 60)], [(257, 250)], [(449, 447)], [(1025, 700)],
    [(40, 50), (17, 9), (90, 80)], [(6 + k % 25, 7 + k % 23) for k in range(330)],
], ids=["one CTA", "a cluster", "clusters", "registers", "pairs", "several", "pieces"])
def test_persistent_cg(shapes):
    check([cloth(c, r, k)[:2] for k, (c, r) in enumerate(shapes)], executor="streamed")


@pytest.mark.parametrize("shapes", [[(15, 14)], [(60, 70)], [(60, 50), (20, 20), (7, 9)]], ids=["one CTA", "one", "several"])
def test_coupled_cg(shapes):
    check([coupled(c, r, k, mode=JAC_COUPLED) for k, (c, r) in enumerate(shapes)])
