"""The refinement in one launch (up to 1,024 unknowns) at the edges of its
blocks and of its range, against numpy and against the separate launches."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(nb, z, b):
    from gpu_helpers import Engine
    e = Engine(nb.lib)
    n = len(b)
    x, res = np.empty(n, dtype=complex), C.c_double(0)
    nb.lib.necgpu_matrix_solve.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    e.check(nb.lib.necgpu_matrix_solve(e.h, n, z.ctypes.data, b.ctypes.data, 1, x.ctypes.data, C.byref(res)))
    its = e.stats().refine_iters
    e.close()
    return x, res.value, its


@pytest.mark.parametrize("n", [2, 63, 64, 65, 129, 511, 1000, 1023, 1024, 1025])
def test_refinement_at_block_edges(nb, monkeypatch, n):
    """A matrix with singular values in [1, 2] (a unitary of a random matrix
    plus half of another): the refined solution is within 1e-12 of numpy's
    (residual tolerance 1e-13, condition at most 3), and both forms of the
    refinement agree and take the same number of steps."""
    rng = np.random.default_rng(n)
    u, v = (np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0] for _ in range(2))
    z = np.ascontiguousarray(1.5 * u + 0.5 * v)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ref = np.linalg.solve(z, b)
    x, res, its = solve(nb, z, b)
    assert res <= 1e-13
    assert np.linalg.norm(x - ref) <= 1e-12 * np.linalg.norm(ref)
    monkeypatch.setenv("NECPP_B200_REFINE_FUSED", "0")
    y, _, its2 = solve(nb, z, b)
    assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(ref)
    assert its == its2
