"""A large general mesh whose Provot pass is turned on and off, which moves its steps between k_sim and
the separate launches: the bits of the streamed executor, for calls of one step and of several."""
import numpy as np
import pytest

from opencloth_gb300 import PASS_PROVOT, ClothSolver
from test_gpu_sim import DT, grid, mesh, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("others", ["none", "some", "many"])
@pytest.mark.parametrize("n", [8000, 9001, 16384])
def test_mixed_calls(n, others):
    """(With "many", beyond 60,000 vertices, calls of several steps stay in k_sim.)"""
    parts = [mesh(n, n)] + {"none": [], "some": [grid(40, 30, 3), mesh(500, 4)], "many": [grid(128, 127, k) for k in range(5)]}[others]
    X, V = np.concatenate([p[1] for p in parts]), np.concatenate([p[2] for p in parts])
    out = []
    for executor in ("auto", "streamed"):
        with ClothSolver([p[0] for p in parts], executor=executor) as s:
            s.set_state(X, V)
            s.step(DT, 1)
            s.set_passes(PASS_PROVOT, 0)
            for k in (1, 2, 1, 1, 3):
                s.step(DT, k)
            s.step(0.5 * DT, 1)
            s.set_passes(0)
            s.step(DT, 1)
            s.step(DT, 2)
            out.append((*s.get_state(), s.stats()[0], s.stats()[2]))
    assert all(same_bits(a, b) for a, b in zip(out[0][:3], out[1][:3]))
    assert np.array_equal(out[0][3], out[1][3]) and np.array_equal(out[0][4], out[1][4])


def test_more_shapes_than_streams():
    """Ten launch shapes: calls of one step take the separate launches, longer ones k_sim."""
    parts = [grid(16 * k + 5, 16, k) for k in range(1, 11)]
    X, V = np.concatenate([p[1] for p in parts]), np.concatenate([p[2] for p in parts])
    out = []
    for executor in ("auto", "streamed"):
        with ClothSolver([p[0] for p in parts], executor=executor) as s:
            s.set_state(X, V)
            for k in (1, 3, 1, 1, 2):
                s.step(DT, k)
            out.append((*s.get_state(), s.stats()[0], s.stats()[2]))
    assert all(same_bits(a, b) for a, b in zip(out[0][:3], out[1][:3]))
    assert np.array_equal(out[0][3], out[1][3]) and np.array_equal(out[0][4], out[1][4])
