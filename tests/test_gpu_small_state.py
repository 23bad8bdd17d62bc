"""oc_set_state, oc_get_state and oc_step_host of handles on both sides of the size up to which the
host checks and moves the arrays itself (16,384 vertices): any subset of the arrays, non-finite
values refused with nothing changed, arrays reused right after the call."""
import numpy as np
import pytest

from opencloth_gb300 import ClothDesc, ClothSolver, OcError, grid_cloth

pytestmark = pytest.mark.gpu
DT = 1.0 / 60.0


@pytest.mark.parametrize("shape", [(3, 3), (21, 21), (128, 128), (5, 3277)])
def test_state(shape):
    X, sp = grid_cloth(*shape, jitter=1e-2)
    n = len(X)
    rng = np.random.default_rng(n)
    A, B, C = (rng.normal(0, 1, (n, 3)).astype(np.float32) for _ in range(3))
    with ClothSolver(ClothDesc(n_vertices=n, springs=sp)) as s:
        s.set_state(A, B, C)
        for a, b in zip(s.get_state(), (A, B, C)):
            assert np.array_equal(a, b)
        s.set_state(V=A)
        s.set_state(C, None, B)  # X and dV
        D = A.copy()
        for k in range(4):  # the array is the caller's again at once
            D[:] = k
            s.set_state(V=D)
        D[:] = np.nan
        for a, b in zip(s.get_state(), (C, np.full_like(A, 3), B)):
            assert np.array_equal(a, b)
        for bad in (np.nan, np.inf, -np.inf):
            for where in ((0, 0), (n - 1, 2)):
                E = A.copy()
                E[where] = bad
                for args in ((E, B, C), (A, E, C), (A, B, E)):
                    with pytest.raises(OcError) as e:
                        s.set_state(*args)
                    assert e.value.status == 3
                with pytest.raises(OcError):
                    s.step_host(E, B.copy(), DT, 1)
        for a, b in zip(s.get_state(), (C, np.full_like(A, 3), B)):
            assert np.array_equal(a, b)
        out = np.empty_like(A)
        s.get_state_into(V=out)
        assert np.array_equal(out, np.full_like(A, 3))


@pytest.mark.parametrize("shape", [(21, 21), (128, 128), (129, 128)])
def test_step_host(shape):
    X, sp = grid_cloth(*shape, jitter=1e-2)
    V = np.random.default_rng(1).normal(0, 0.1, X.shape).astype(np.float32)
    d = ClothDesc(n_vertices=len(X), springs=sp, pinned=np.array([0], np.int32))
    with ClothSolver(d) as s, ClothSolver(d) as t:
        for h in (s, t):
            h.set_state(X, V, np.zeros_like(X))
        a, b = X.copy(), V.copy()
        for n in (1, 0, 3):
            s.step_host(a, b, DT, n)
            t.step(DT, n)
        s.step_host(None, b, DT, 1)
        t.step(DT, 1)
        for x, y in zip(s.get_state(), t.get_state()):
            assert np.array_equal(x, y)
        assert np.array_equal(b, t.get_state()[1])


@pytest.mark.parametrize("n", [9, 255, 256, 257, 1023, 40000])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_state_out_to_device_arrays(n, offset):
    """k_state_out4 (16-byte aligned arrays) and k_state_out, in whole blocks and remainders, with
    nothing written beyond the arrays."""
    torch = pytest.importorskip("torch")
    _, sp = grid_cloth(3, 3)
    rng = np.random.default_rng(n)
    A = [rng.normal(0, 1, (n, 3)).astype(np.float32) for _ in range(3)]
    with ClothSolver(ClothDesc(n_vertices=n, springs=sp)) as s:
        s.set_state(*A)
        for given in ((0, 1, 2), (0,), (1, 2), (2,)):
            out = [torch.full((3 * n + 16,), 7.0, device="cuda") for _ in range(3)]
            torch.cuda.synchronize()
            s.get_state_device(*(out[k].data_ptr() + 4 * offset if k in given else 0 for k in range(3)))
            s.synchronize()
            for k in range(3):
                o = out[k].cpu().numpy()
                want = np.full(3 * n + 16, 7.0, np.float32)
                if k in given:
                    want[offset:offset + 3 * n] = A[k].ravel()
                assert np.array_equal(o, want)
