"""The resident FEM CG at the edges of its layout: row counts around warps and the largest CTA,
rows without blocks, the longest rows, fixed rows anywhere, several sizes in one launch.  Its FP32
row arithmetic is the streamed executor's in the same order and its scalars differ only beyond
their floats' digits, so the same bits are expected."""
import numpy as np
import pytest

from opencloth_gb300.fem import BsrSolver

pytestmark = pytest.mark.gpu


def system(n, seed, most=12, fixed=0.15, i_max=12):
    rng = np.random.default_rng(seed)
    cols, rows = [], [0]
    for r in range(n):
        k = 0 if n > 4 and r % 11 == 5 else int(rng.integers(1, min(n, most) + 1))
        c = np.sort(rng.choice(n, k, replace=False))
        if k and r not in c:
            c = np.unique(np.append(c[:-1], r))
        cols.append(c)
        rows.append(rows[-1] + len(c))
    col = np.concatenate(cols).astype(np.int32)
    row = np.repeat(np.arange(n), np.diff(rows))
    blocks = rng.normal(0, 0.02, (len(col), 3, 3))
    blocks[row == col] += np.eye(3) * rng.uniform(1, 2, ((row == col).sum(), 1, 1))
    return {"row_ptr": np.array(rows, np.int32), "col": col, "blocks": blocks.reshape(-1, 9).astype(np.float32),
            "b": rng.normal(0, 1, (n, 3)).astype(np.float32), "V": rng.normal(0, 1, (n, 3)).astype(np.float32),
            "fixed": (rng.random(n) < fixed).astype(np.uint8), "i_max": i_max, "tolerance": 1e-3, "tiny": 1e-10}


def solve(systems, executor):
    with BsrSolver(systems, executor=executor) as s:
        s.set_system(*(np.concatenate([g[k] for g in systems]) for k in ("blocks", "b", "V")))
        s.solve()
        return s.solution()


@pytest.mark.parametrize("n,most", [(1, 1), (2, 2), (31, 8), (32, 32), (33, 5), (64, 64), (176, 19), (255, 16), (256, 12)])
def test_sizes(n, most):
    systems = [system(n, 7 * n + k, most) for k in range(3)]
    for a, b in zip(solve(systems, 2), solve(systems, 1)):
        assert np.array_equal(a, b)


def test_mixed_sizes_and_all_fixed():
    systems = [system(40, 1), system(200, 2, 20), system(90, 3, fixed=1.0), system(5, 4, i_max=0), system(256, 5, 4)]
    for a, b in zip(solve(systems, 2), solve(systems, 1)):
        assert np.array_equal(a, b)
