"""Blocked solves with many right-hand sides at the edges of their output tiles
(16 and 64 rows, 64 right-hand sides) and on both sides of the line between them."""
import numpy as np
import pytest

from test_gpu_mixed import backward_error, mixed_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrhs", [(130, 17), (641, 64), (641, 65), (1025, 129), (1600, 770)])
def test_right_hand_sides_reach_the_gate(gpu_lib, n, nrhs):
    rng = np.random.default_rng(n)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 2 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
    s, X, be, it = mixed_solve(gpu_lib, Z, B)
    assert s == 0, (be, it)
    for q in (0, 1, nrhs // 2, nrhs - 1):
        assert backward_error(Z, X[q], B[q]) <= 1e-10
