"""The FP64 panel in one cluster at the edges of its blocks and of its range."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(nb):
    from gpu_helpers import Engine
    e = Engine(nb.lib)
    nb.lib.necgpu_matrix_solve.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    yield e
    e.close()


def solve(nb, e, z, b):
    x = np.empty(len(b), dtype=complex)
    rc = nb.lib.necgpu_matrix_solve(e.h, len(b), z.ctypes.data, b.ctypes.data, 0, x.ctypes.data, None)
    return rc, x


# one panel (whole and partial blocks of eight columns), several, a row per
# CTA and the most the cluster holds (3,296), one more than that
@pytest.mark.parametrize("n", [1, 7, 8, 9, 63, 64, 65, 71, 128, 517, 1040, 3296, 3297])
def test_fp64_solve_at_panel_edges(nb, engine, n):
    """Rows of a random matrix shuffled and scaled by up to 1e6, so that most
    columns exchange rows: backward error ||b - Z x|| / (||Z|| ||x||) below
    n eps (partial pivoting's is a few eps on random matrices)."""
    if n == 1:
        z, b = np.array([[2.0 - 1.0j]]), np.array([1.0 + 3.0j])
    else:
        rng = np.random.default_rng(n)
        z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        z = np.ascontiguousarray(z * 10.0 ** rng.uniform(0.0, 6.0, (n, 1)))
        b = (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * np.abs(z).max(axis=1)
    rc, x = solve(nb, engine, z, b)
    assert rc == 0, engine.err()
    r = np.abs(b - z @ x)
    assert np.max(r / (np.abs(z) @ np.abs(x))) <= max(n, 8) * 2.3e-16


@pytest.mark.parametrize("value,code", [(0.0, 3), (float("nan"), 4)])
def test_fp64_panel_bad_column(nb, engine, value, code):
    """A column of zeros is reported as singular, one of NaNs as non-finite."""
    rng = np.random.default_rng(4)
    z = rng.standard_normal((100, 100)) + 1j * rng.standard_normal((100, 100))
    z[:, 70] = value
    rc, _ = solve(nb, engine, z, np.ones(100, dtype=complex))
    assert rc == code
