"""The largest systems of the resident FEM CG (executor 2): what 37 bytes a block in one CTA's shared
memory hold, 6,088 blocks with 256 rows, is accepted and gives the streamed executor's bits; more is refused."""
import numpy as np
import pytest

from opencloth_gb300 import OcError
from opencloth_gb300.fem import BsrSolver
from test_gpu_fem_resident import solve

pytestmark = pytest.mark.gpu


def system(nnzb, fixed=0.0, n=256, longest=64, i_max=9):
    """n rows of nnzb blocks together, the first of `longest`."""
    rng = np.random.default_rng(nnzb)
    deg = np.full(n, (nnzb - longest) // (n - 1))
    deg[0] = longest
    deg[1:1 + nnzb - deg.sum()] += 1
    assert deg.sum() == nnzb and deg.max() <= 64
    cols = [np.sort(np.append(rng.choice(np.setdiff1d(np.arange(n), [r]), deg[r] - 1, replace=False), r)) for r in range(n)]
    col = np.concatenate(cols).astype(np.int32)
    row = np.repeat(np.arange(n), deg)
    blocks = rng.normal(0, 0.01, (nnzb, 3, 3))
    blocks[row == col] += np.eye(3) * rng.uniform(1, 2, (n, 1, 1))
    return {"row_ptr": np.append(0, np.cumsum(deg)).astype(np.int32), "col": col,
            "blocks": blocks.reshape(-1, 9).astype(np.float32), "b": rng.normal(0, 1, (n, 3)).astype(np.float32),
            "V": rng.normal(0, 1, (n, 3)).astype(np.float32), "fixed": (rng.random(n) < fixed).astype(np.uint8),
            "i_max": i_max, "tolerance": 1e-3, "tiny": 1e-10}


@pytest.mark.parametrize("nnzb,fixed", [(5600, 0.0), (5700, 0.0), (6000, 0.2), (6088, 0.0), (6088, 0.3)])
def test_accepted(nnzb, fixed):
    systems = [system(nnzb, fixed), system(3000, 0.1, n=180), system(nnzb - 40, 0.0)]
    for a, b in zip(solve(systems, 2), solve(systems, 1)):
        assert np.array_equal(a, b)
    for a, b in zip(solve(systems, 0), solve(systems, 1)):
        assert np.array_equal(a, b)


def test_refused():
    with pytest.raises(OcError) as e:
        BsrSolver([system(6089)], executor=2)
    assert e.value.status == 7


@pytest.mark.parametrize("nnzb", [5000, 6000])
def test_a_smaller_handle_made_later(nnzb):
    """Its shared memory is no limit for the larger handle's solves."""
    large, small = system(nnzb), system(1400, n=100, longest=20)
    want = solve([large], 1)
    with BsrSolver([large], executor=2) as s:
        with BsrSolver([small], executor=2):
            s.set_system(large["blocks"], large["b"], large["V"])
            s.solve()
            assert all(np.array_equal(a, b) for a, b in zip(s.solution(), want))
