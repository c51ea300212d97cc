"""Trailing updates of the FP64 LU on the tensor cores (integer digits,
digit_gemm.cu) at the edges of their blocks and tiles (64-column blocks,
128-row and 48 / 96-column tiles).

The factor is checked by its componentwise backward error |P A - L U| <= c n u
|L| |U| (Higham, Accuracy and Stability of Numerical Algorithms, theorem 9.3:
gamma_n for real arithmetic, 2 sqrt(2) gamma_n-like for complex), formed in
extended precision on sampled rows."""
import math

import numpy as np
import pytest

from helpers import ComplexLU, RealLU

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def matrix(n, cplx, kind):
    rng = np.random.default_rng(1000 + n)
    a = rng.standard_normal((n, n))
    if cplx:
        a = a + 1j * rng.standard_normal((n, n))
    if kind == "decaying":  # 1/distance-like rows of widely different size
        i = np.arange(n)
        a = a / (1.0 + np.abs(i[:, None] - i[None])) ** 2 * np.logspace(-6, 6, n)[:, None]
    return a


def factored(lib, a, cplx):
    f = ComplexLU(lib, a) if cplx else RealLU(lib, a)
    assert f.status == 0
    if cplx:
        lu, piv, rs, cs = f.factors()
    else:
        lu, piv = f.factors()
        rs = cs = np.ones(len(a))
    f.free()
    return lu, piv, rs, cs


def permuted(a, piv):
    a = a.copy()
    for k, p in enumerate(piv):
        if p != k:
            a[[k, p]] = a[[p, k]]
    return a


def backward_error(a, lu, piv, rs, cs, cplx, rows):
    """max |P A - L U| / (|L| |U|) over the sampled rows, products in extended precision."""
    n = len(a)
    ld = np.clongdouble if cplx else np.longdouble
    scaled = (a / rs[:, None]) / cs[None, :] if cplx else a
    pa = permuted(scaled, piv)
    worst = 0.0
    Uu = np.triu(lu).astype(ld)
    for i in rows:
        li = np.zeros(n, dtype=ld)
        li[:i], li[i] = lu[i, :i], 1
        e = np.abs(li @ Uu - pa[i].astype(ld))
        w = np.abs(li).astype(np.longdouble) @ np.abs(Uu).astype(np.longdouble)
        worst = max(worst, float(np.max(np.where(w > 0, e / np.where(w > 0, w, 1), e))))
    return worst


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [64, 65, 127, 128, 129, 191, 193, 257, 451])
@pytest.mark.parametrize("kind", ["normal", "decaying"])
def test_backward_error_at_block_edges(gpu_lib, n, cplx, kind):
    a = matrix(n, cplx, kind)
    lu, piv, rs, cs = factored(gpu_lib, a, cplx)
    rows = sorted({0, 1, 63, 64, 65, n // 2, n - 2, n - 1} & set(range(n)))
    # gamma_n for real, 2 sqrt(2) gamma_n + the scaling's two divisions for complex
    bound = (2 * math.sqrt(2) * n + 4) * U if cplx else n * U / (1 - n * U)
    assert backward_error(a, lu, piv, rs, cs, cplx, rows) <= bound


def test_pivots_match_the_oracle_over_several_blocks(gpu_lib, oracle):
    for n in (130, 200, 333):
        a = matrix(n, True, "normal")
        _, piv, _, _ = factored(gpu_lib, a, True)
        assert np.array_equal(piv, oracle.complex_lu_factorize(a)[2].astype(np.int64))


def test_columns_of_widely_different_size(gpu_lib):
    """Columns scaled by powers of two from 2^-280 to 2^280: the pivots are those
    of the unscaled matrix (a column's scale changes none of its comparisons),
    and the backward error keeps its bound."""
    n = 300
    a = matrix(n, False, "normal")
    rng = np.random.default_rng(4)
    d = np.ldexp(1.0, rng.integers(-280, 281, n))
    lu0, piv0, _, _ = factored(gpu_lib, a, False)
    lu1, piv1, _, _ = factored_low_tolerance(gpu_lib, a * d[None, :])
    assert np.array_equal(piv0, piv1)
    rows = [0, 63, 64, 65, 150, 298, 299]
    # (the extended-precision check works on the unscaled columns)
    lu1 = np.tril(lu1, -1) + np.triu(lu1) / d[None, :]
    assert backward_error(a, lu1, piv1, np.ones(n), np.ones(n), False, rows) <= n * U / (1 - n * U)


@pytest.mark.parametrize("eps", [1e-7, 1e-12, 1e-20])
def test_weakly_coupled_parts(gpu_lib, eps):
    """Two interleaved sets of unknowns coupled by entries eps times the others:
    the coupling's entries keep their own relative accuracy (they are far below
    their rows' and columns' sizes and take the FP64 chain)."""
    n = 320
    a = matrix(n, True, "normal")
    i = np.arange(n) % 2
    a = np.where(i[:, None] == i[None, :], a, a * eps)
    lu, piv, rs, cs = factored(gpu_lib, a, True)
    rows = [1, 64, 65, 127, 128, 200, 318, 319]
    assert backward_error(a, lu, piv, rs, cs, True, rows) <= (2 * math.sqrt(2) * n + 4) * U


@pytest.mark.parametrize("n", [3001, 3200])
def test_wide_outer_blocks(gpu_lib, n):
    """From 3000 unknowns on the outer blocks are wider than the inner ones
    (192 columns complex, 256 real): ragged last blocks of both kinds."""
    for cplx in (False, True):
        a = matrix(n, cplx, "decaying")
        lu, piv, rs, cs = factored(gpu_lib, a, cplx)
        rows = [0, 191, 192, 255, 256, n // 2, n - 2, n - 1]
        bound = (2 * math.sqrt(2) * n + 4) * U if cplx else n * U / (1 - n * U)
        assert backward_error(a, lu, piv, rs, cs, cplx, rows) <= bound


def factored_low_tolerance(lib, a):
    f = RealLU(lib, a, tol=1e-300)
    assert f.status == 0
    lu, piv = f.factors()
    f.free()
    return lu, piv, None, None


def test_columns_of_zeros_and_subnormals(gpu_lib):
    """Zero columns of the trailing block's multipliers and entries far below
    their row's largest leave C as it is."""
    n = 192
    rng = np.random.default_rng(8)
    a = np.triu(rng.standard_normal((n, n))) + 4 * np.eye(n)  # L = I: every update subtracts zero
    lu, piv, _, _ = factored(gpu_lib, a, False)
    assert np.array_equal(piv, np.arange(n)) and np.array_equal(lu, a)
    b = a.copy()
    b[100:, 3] = 5e-320  # subnormal multipliers: products far below the entries
    lu, piv, _, _ = factored(gpu_lib, b, False)
    assert np.array_equal(piv, np.arange(n))
    assert np.array_equal(np.triu(lu), np.triu(a))


def test_tied_rows_give_the_oracles_pivots(gpu_lib, oracle):
    """Rows in pairs that agree in their first 300 columns and in the last one,
    whose entry is the largest of the row (so the equilibration keeps the pairs
    equal): in each of those columns the two copies tie exactly and the lower row
    wins, as in the oracle."""
    n, m = 1400, 300
    rng = np.random.default_rng(12)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    a[:, -1] = 64.0 * (1.0 + rng.random(n))
    a[n // 2:, :m] = a[:n // 2, :m]
    a[n // 2:, -1] = a[:n // 2, -1]
    _, piv, _, _ = factored(gpu_lib, a, True)
    assert np.array_equal(piv, oracle.complex_lu_factorize(a)[2].astype(np.int64))


@pytest.mark.parametrize("n,cplx", [(n, c) for n in (33, 63, 95, 97) for c in (False, True)] + [(1313, True), (1345, True)])
def test_ragged_columns_right_of_a_block(gpu_lib, n, cplx):
    """Rows of U are solved in tiles of 32 columns, 32 rows at once in small
    systems and 64 in large ones: last tiles of 1, 31 and 33 columns."""
    a = matrix(n, cplx, "normal")
    lu, piv, rs, cs = factored(gpu_lib, a, cplx)
    rows = sorted({0, 7, 8, 31, 32, 63, n // 2, n - 1} & set(range(n)))
    bound = (2 * math.sqrt(2) * n + 4) * U if cplx else n * U / (1 - n * U)
    assert backward_error(a, lu, piv, rs, cs, cplx, rows) <= bound
