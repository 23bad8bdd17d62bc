"""The persistent CG's plans (oc_persist.cu) at the edges of what a CTA holds in registers, in
shared memory and in the planes: each against the two-kernel WHILE loop (OC_PERSIST=0), whose
sums differ from it only beyond the digits that alpha, beta and the stop test keep, so the same
bits, iteration counts and flags are expected."""
import numpy as np
import pytest

from test_gpu_persist import cloth, run, same_bits

pytestmark = pytest.mark.gpu

# With 256 threads a CTA and 112 CTAs in clusters of 16: one vertex a thread up to 28,672
# vertices, everything in registers up to 7 (200,704), x beside A, r and d on chip up to 28
# slots or so; beyond that all SMs in clusters of 2, and past a million vertices slots that stay
# in the planes.
SIZES = [(9, 7), (16, 16), (257, 3), (64, 64), (167, 172), (169, 170), (251, 229), (401, 501), (449, 447), (811, 901),
         (1025, 1023), (1300, 1009)]


@pytest.mark.parametrize("cols,rows", SIZES, ids=lambda v: str(v))
def test_one_cloth(cols, rows):
    d, X, V = cloth(cols, rows, cols + rows)
    a, sa = run(d, X, V, 2, True, executor="streamed")
    b, sb = run(d, X, V, 2, False, executor="streamed")
    for x, y in zip(a, b):
        assert same_bits(x, y)
    assert np.array_equal(sa[0], sb[0]) and np.array_equal(sa[2], sb[2]) and sa[0][0] > 0


@pytest.mark.parametrize("strip", [0, 1])
@pytest.mark.parametrize("count,lo,hi", [(5, 8, 90), (112, 8, 40), (113, 8, 40), (330, 6, 30), (9, 120, 260)])
def test_several_cloths(count, lo, hi, strip):
    """Up to as many cloths as CTAs (each CTA one piece), and more (several pieces a CTA, cloths
    that share a cluster's CTAs), with and without the strip sweep's delta0."""
    import os

    rng = np.random.default_rng(count)
    parts = [cloth(int(rng.integers(lo, hi + 1)), int(rng.integers(lo, hi + 1)), 700 + k,
                   ks=tuple(np.exp(rng.uniform(np.log(10.0), np.log(500.0), 3)))) for k in range(count)]
    descs = [p[0] for p in parts]
    X, V = np.concatenate([p[1] for p in parts]), np.concatenate([p[2] for p in parts])
    old = os.environ.get("OC_STRIP")
    os.environ["OC_STRIP"] = str(strip)
    try:
        a, sa = run(descs, X, V, 3, True, executor="streamed")
        b, sb = run(descs, X, V, 3, False, executor="streamed")
    finally:
        os.environ.pop("OC_STRIP")
        if old is not None:
            os.environ["OC_STRIP"] = old
    for x, y in zip(a, b):
        assert same_bits(x, y)
    assert np.array_equal(sa[0], sb[0]) and np.array_equal(sa[2], sb[2])
