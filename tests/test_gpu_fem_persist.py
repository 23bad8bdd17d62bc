"""The streamed FEM CG in one cooperative launch (k_bsr_persist) against the same solve launch by
launch (use_graph=False): the same row arithmetic in the same order, scalars that differ only beyond
their floats' digits, so the same bits.  Sizes around a CTA's rows, rows beyond one per thread,
several systems side by side, and more systems than SMs (the WHILE loop)."""
import numpy as np
import pytest

from opencloth_gb300.fem import BsrSolver, fem_system
from test_gpu_fem_resident import system

pytestmark = pytest.mark.gpu


def solve(systems, **kw):
    with BsrSolver(systems, executor=1, **kw) as s:
        s.set_system(*(np.concatenate([g[k] for g in systems]) for k in ("blocks", "b", "V")))
        s.solve()
        first = s.solution()
        s.set_system(None, np.concatenate([g["b"] for g in systems]), np.concatenate([g["V"] for g in systems]))
        s.solve()  # new vectors, the blocks kept
        again = s.solution()
    assert all(np.array_equal(a, b) for a, b in zip(first, again))
    return first


def check(systems):
    for a, b in zip(solve(systems), solve(systems, use_graph=False)):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("n", [1, 33, 256, 257, 1000, 3000])
@pytest.mark.parametrize("i_max", [0, 1, 7])
def test_one_system(n, i_max):
    check([system(n, n, 9, i_max=i_max)])


def test_several_systems_of_different_lengths():
    check([system(300, 1, i_max=3), system(2100, 2, 15), system(40, 3, fixed=1.0), system(700, 4, 30, i_max=9)])


@pytest.mark.parametrize("count", [100, 170])
def test_many_systems(count):
    check([system(30 + k % 50, k, 6, i_max=1 + k % 5) for k in range(count)])


def test_rows_beyond_one_per_thread():
    n = 65 * 51 * 51  # more than 1,024 rows on each of 152 SMs
    check([fem_system(64, 50, 50, V=np.random.default_rng(2).normal(0, 0.1, (n, 3)), i_max=5)])
