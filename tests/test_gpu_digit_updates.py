"""The digit GEMM by itself (peec_gb300_digit_gemm_sub) at the edges of its tiles
(128 rows, 48 complex or 96 real columns, 16 of K), the LU with its form of the
updates given, and the inverse of a transient system with digits.

An update is C - sum rounded twice: u |sum| + u |C - sum|, and what is dropped
of the digits: pairs i + j >= 14 of 12 digits of at most 64 in units 2^-7, 11 of
them with i + j = 14, 2 K products each (K <= 192 complex, K <= 256 real), in all below
2^-71.8 of the scales of row and column, which are less than twice their 2-norms
(the inner scaling by the exponents of B's rows included).  Entries that take
FP64 FMAs are within gamma_2K of the sum of magnitudes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
TURNS = np.array([1, 1j, -1, -1j])


class Device:
    """Device copies of host arrays, freed together."""

    def __init__(self, lib):
        self.lib, self.p = lib, []

    def __enter__(self):
        return self

    def __exit__(self, *_):
        for p in self.p:
            self.lib.peec_gb300_device_free(p)

    def put(self, a):
        p = self.lib.peec_gb300_device_alloc(max(a.nbytes, 16))
        self.p.append(p)
        assert self.lib.peec_gb300_copy_to_device(p, a.ctypes.data, a.nbytes) == 0
        return p

    def get(self, p, like):
        out = np.empty_like(like)
        assert self.lib.peec_gb300_copy_to_host(out.ctypes.data, p, out.nbytes) == 0
        return out


def digit_sub(lib, a, b, c, pad=(0, 0, 0), skip=0):
    """C - A B by the library; pad: extra columns of A, B, C in memory; skip: entries before C."""
    cplx = a.dtype == np.complex128
    wide = [np.pad(x, ((0, 0), (0, e)), constant_values=7.0) for x, e in zip((a, b, c), pad)]
    flat = np.concatenate([np.zeros(skip, dtype=c.dtype), wide[2].ravel()])
    size = flat.itemsize
    with Device(lib) as d:
        pa, pb, pc = d.put(wide[0]), d.put(wide[1]), d.put(flat)
        assert lib.peec_gb300_digit_gemm_sub(int(cplx), pa, wide[0].shape[1], pb, wide[1].shape[1], pc + skip * size,
                                             wide[2].shape[1], *c.shape, a.shape[1]) == 0
        out = d.get(pc, flat)
    assert np.array_equal(out[:skip], flat[:skip])
    out = out[skip:].reshape(wide[2].shape)
    assert np.array_equal(out[:, c.shape[1]:], wide[2][:, c.shape[1]:])
    return out[:, :c.shape[1]]


def parts(x):
    return (x.real, x.imag) if np.iscomplexobj(x) else (x,)


def sums(a, b, rows):
    """A B on the given rows by parts, in extended precision, and the sums of magnitudes."""
    ld = np.longdouble
    a = [p[rows].astype(ld) for p in parts(a)]
    b = [p.astype(ld) for p in parts(b)]
    if len(a) == 1:
        return [a[0] @ b[0]], [abs(a[0]) @ abs(b[0])]
    return ([a[0] @ b[0] - a[1] @ b[1], a[0] @ b[1] + a[1] @ b[0]],
            [abs(a[0]) @ abs(b[0]) + abs(a[1]) @ abs(b[1]), abs(a[0]) @ abs(b[1]) + abs(a[1]) @ abs(b[0])])


def exponent(x):
    """Powers of two above |x| (1 for zeros)."""
    return np.where(x > 0, np.exp2(np.floor(np.log2(np.where(x > 0, x, 1.0))) + 1), 1.0)


def scales(a, b):
    """The scales of rows and columns are below twice these 2-norms."""
    f = exponent(np.max([abs(p).max(axis=1) for p in parts(b)], axis=0))
    return np.linalg.norm(a * f[None], axis=1), np.linalg.norm(b / f[:, None], axis=0)


def check(a, b, c, out, rows, floor=True):
    """floor: the digits' absolute error is allowed beside that of the FP64 operations."""
    k = a.shape[1]
    exact, mags = sums(a, b, rows)
    ra, cb = scales(a, b)
    dropped = 2.0 ** -71.8 * 4 * ra[rows][:, None] * cb[None] if floor else 0.0
    gamma = 2 * k * U / (1 - 2 * k * U)
    for e, w, x, y in zip(exact, mags, parts(c), parts(out)):
        want = x[rows].astype(np.longdouble) - e
        err = abs(y[rows].astype(np.longdouble) - want)
        assert np.all(err <= gamma * w + 1.01 * U * abs(want) + dropped)
        if floor:  # digits: rounded twice; the bound of FMA chains only below 2^-25 of the scales
            tight = 1.01 * U * (abs(e) + abs(want)) + dropped
            line = 2.0 ** -24 * 4 * ra[rows][:, None] * cb[None]
            assert np.all(err <= np.where((abs(e) < line) & (abs(x[rows]) < line), gamma * w + tight, tight))


def normal(rng, cplx, *shape):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


def some(m):
    return sorted({0, 1, 31, 32, 63, 127, 128, 129, m - 1} & set(range(m)))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,k,pad,skip", [
    (1, 1, 1, (0, 0, 0), 0), (127, 47, 15, (0, 0, 0), 1), (128, 48, 16, (1, 1, 1), 0), (129, 49, 17, (3, 0, 5), 3),
    (128, 96, 64, (0, 0, 0), 0), (130, 97, 63, (0, 2, 1), 1), (257, 95, 65, (0, 0, 0), 0), (64, 193, 128, (0, 0, 3), 0),
    (129, 145, 129, (0, 1, 0), 1), (300, 33, 191, (0, 0, 0), 0), (40, 290, 192, (0, 0, 0), 0), (200, 100, 256, (0, 0, 1), 1)])
def test_edges_of_tiles(gpu_lib, cplx, m, n, k, pad, skip):
    if cplx and k > 192:
        k = 192
    rng = np.random.default_rng(m + 1000 * n + k)
    a, b, c = normal(rng, cplx, m, k), normal(rng, cplx, k, n), normal(rng, cplx, m, n)
    check(a, b, c, digit_sub(gpu_lib, a, b, c, pad, skip), some(m))


def test_more_tiles_than_ctas(gpu_lib):
    """Each CTA takes several tiles: 8 x 32 complex ones and 16 x 16 real ones."""
    for cplx, m, n, k in ((True, 1000, 1530, 80), (False, 2000, 1530, 100)):
        rng = np.random.default_rng(3)
        a, b, c = normal(rng, cplx, m, k), normal(rng, cplx, k, n), normal(rng, cplx, m, n)
        check(a, b, c, digit_sub(gpu_lib, a, b, c), [0, 127, 128, 500, 640, m - 1])


@pytest.mark.parametrize("cplx", [False, True])
def test_scales_of_rows_columns_and_inner_index(gpu_lib, cplx):
    """Powers of two change nothing but the scale of the result."""
    m, n, k = 140, 100, 70
    rng = np.random.default_rng(5)
    a, b, c = normal(rng, cplx, m, k), normal(rng, cplx, k, n), normal(rng, cplx, m, n)
    plain = digit_sub(gpu_lib, a, b, c)
    r, s, t = (np.ldexp(1.0, rng.integers(-200, 201, x)) for x in (m, n, k))
    scaled = digit_sub(gpu_lib, a * r[:, None] * t[None], b / t[:, None] * s[None], c * r[:, None] * s[None])
    assert np.array_equal(scaled / r[:, None] / s[None], plain)


@pytest.mark.parametrize("cplx", [False, True])
def test_zeros_subnormals_and_coherent_digits(gpu_lib, cplx):
    m, n, k = 135, 99, 192
    rng = np.random.default_rng(6)
    a, b, c = normal(rng, cplx, m, k), normal(rng, cplx, k, n), normal(rng, cplx, m, n)
    a[3], b[:, 5], a[:, 9], b[11] = 0, 0, 0, 0
    a[130, ::2] = 5e-320
    # equal 53-bit entries of alternating signs: every digit pair adds up the same way
    x = 1.0 + 63.0 / 127.0  # all digits 63
    a[40] = np.where(np.arange(k) % 2, x, -x)
    b[:, 60] = np.where(np.arange(k) % 2, x, -x) if not cplx else np.where(np.arange(k) % 2, x, -x) * (1 + 1j)
    a[41] = x
    out = digit_sub(gpu_lib, a, b, c)
    check(a, b, c, out, [0, 3, 40, 41, 130, 134])
    assert np.array_equal(out[3], c[3]) and np.array_equal(out[:, 5], c[:, 5])


@pytest.mark.parametrize("cplx", [False, True])
def test_infinities_and_nans(gpu_lib, cplx):
    """Only the rows and columns that hold them are touched, as in FP64."""
    m, n, k = 140, 100, 40
    rng = np.random.default_rng(7)
    a, b, c = normal(rng, cplx, m, k), normal(rng, cplx, k, n), normal(rng, cplx, m, n)
    a[2, 3], a[133, 39], b[0, 97], b[17, 1] = np.nan, np.inf, np.inf, np.nan
    c[50, 50] = np.inf
    out = digit_sub(gpu_lib, a, b, c)
    bad = np.zeros((m, n), dtype=bool)
    bad[[2, 133]] = bad[:, [97, 1]] = True
    bad[50, 50] = True
    assert np.array_equal(~np.isfinite(out), bad)
    a[~np.isfinite(a)], b[~np.isfinite(b)], c[50, 50] = 0, 0, 0
    ok = ~bad
    rows = [0, 49, 128, 139]
    exact, _ = sums(a, b, rows)
    for e, x, y in zip(exact, parts(c), parts(out)):
        assert np.all(abs(y[rows] - (x[rows] - e))[ok[rows]] <= 4 * U * (abs(e) + abs(x[rows]))[ok[rows]] + 1e-20)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("every", [2, 40])
@pytest.mark.parametrize("eps", [1e-9, 1e-20])
def test_entries_far_below_their_rows_and_columns(gpu_lib, cplx, every, eps):
    """Rows and columns in two sets, coupled by eps: the coupled entries take
    FP64 FMAs, half of a warp's lanes at once or one lane at a time."""
    m, n, k = 200, 150, 128
    rng = np.random.default_rng(8)
    i, j, q = np.arange(m) % every == 0, np.arange(n) % every == 0, np.arange(k) % 2 == 0
    a = normal(rng, cplx, m, k) * np.where(i[:, None] == q[None], 1.0, eps)
    b = normal(rng, cplx, k, n) * np.where(q[:, None] == j[None], 1.0, eps)
    c = normal(rng, cplx, m, n) * np.where(i[:, None] == j[None], 1.0, eps)
    check(a, b, c, digit_sub(gpu_lib, a, b, c), [0, 1, 39, 40, 80, 81, 198, 199], floor=False)


# ---- LU with the form of its updates given -----------------------------------------
FMA, DIGITS, CHECKED = 0, 1, 2


def factor(lib, a, form, tol=1e-14):
    """status, factor, pivots, row and column scales, form that was used"""
    n, cplx = len(a), a.dtype == np.complex128
    a = np.ascontiguousarray(a)
    with Device(lib) as d:
        p = [d.put(a), d.put(np.zeros(n, np.int64)), d.put(np.zeros(n, np.int32)), d.put(np.ones(n)), d.put(np.ones(n))]
        used = C.c_int(-1)
        s = lib.peec_gb300_lu_factor_device_form(int(cplx), p[0], n, tol, p[1], p[2], p[3] if cplx else None,
                                                 p[4] if cplx else None, form, C.byref(used))
        like = (a, np.zeros(n, np.int64), np.ones(n), np.ones(n))
        return (s, *[d.get(x, y) for x, y in zip((p[0], p[1], p[3], p[4]), like)], used.value)


def residual(a, lu, piv, rs, cs):
    """|P A - L U| / (|L| |U|) on a few rows (extended precision)"""
    n = len(a)
    ld = np.clongdouble if np.iscomplexobj(a) else np.longdouble
    pa = (a / rs[:, None]) / cs[None]
    for k, p in enumerate(piv):
        if p != k:
            pa[[k, p]] = pa[[p, k]]
    worst, up = 0.0, np.triu(lu).astype(ld)
    for i in sorted({0, 63, 64, 65, 129, 191, 192, 255, 256, n // 2, n - 2, n - 1} & set(range(n))):
        li = np.zeros(n, dtype=ld)
        li[:i], li[i] = lu[i, :i], 1
        worst = max(worst, float(np.max(abs(li @ up - pa[i]) / (abs(li) @ abs(up)))))
    return worst


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [65, 128, 129, 193, 257, 451])
@pytest.mark.parametrize("form", [DIGITS, CHECKED])
def test_lu_by_digits_at_block_edges(gpu_lib, n, cplx, form):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    for decay in (0, 2):
        a = normal(rng, cplx, n, n) / (1.0 + abs(i[:, None] - i[None])) ** decay
        s, lu, piv, rs, cs, used = factor(gpu_lib, a, form)
        assert s == 0 and used == 1
        bound = (2 * np.sqrt(2) * n + 4) * U if cplx else n * U / (1 - n * U)
        assert residual(a, lu, piv, rs, cs) <= bound
        assert np.array_equal(piv, factor(gpu_lib, a, FMA)[2])


@pytest.mark.parametrize("cplx,n", [(False, 6273), (True, 5601)])
def test_lu_by_digits_in_wide_blocks(gpu_lib, cplx, n):
    """Outer blocks of 256 real (from 6200 unknowns) and 192 complex columns (from 5500),
    the last one ragged: P A x = L U x for signs x, each side within gamma_n |L| |U| |x|
    of the exact one, twice that for L U x and once for the factor."""
    a = normal(np.random.default_rng(1), cplx, n, n)
    s, lu, piv, rs, cs, used = factor(gpu_lib, a, CHECKED)
    assert s == 0 and used == 1
    a = (a / rs[:, None]) / cs[None]
    order = np.arange(n)
    for k, p in enumerate(piv):
        order[[k, p]] = order[[p, k]]
    l, u = np.tril(lu, -1), np.triu(lu)
    x = np.random.default_rng(2).choice([-1.0, 1.0], (n, 4))
    y, z = u @ x, np.abs(u) @ np.abs(x)
    gamma = (2 * np.sqrt(2) if cplx else 1.0) * n * U / (1 - n * U)
    assert np.all(abs(l @ y + y - (a @ x)[order]) <= 4 * gamma * (np.abs(l) @ z + z))


def test_complex_sizes_that_take_digits_by_themselves(gpu_lib):
    """From 1300 complex unknowns on the factorisation is the checked one, bit for bit."""
    n = 1313
    a = normal(np.random.default_rng(2), True, n, n)
    s, lu, piv, _, _, used = factor(gpu_lib, a, CHECKED)
    assert s == 0 and used == 1
    with Device(gpu_lib) as d:
        p = [d.put(a), d.put(np.zeros(n, np.int64)), d.put(np.zeros(n, np.int32)), d.put(np.ones(n)), d.put(np.ones(n))]
        assert gpu_lib.peec_gb300_complex_lu_factor_device(p[0], n, 1e-14, *p[1:], None, None) == 0
        assert np.array_equal(d.get(p[0], a), lu) and np.array_equal(d.get(p[1], piv), piv)


@pytest.mark.parametrize("n", [64, 65, 999, 1000, 1025, 1300, 2049])
def test_inverse(gpu_lib, n):
    """Digits from 1000 unknowns on, outer blocks of 256: the blocked substitution
    keeps |L U X - P| <= 2 gamma_n |L| |U| |X| (twice that for the check's own FP64)."""
    a = normal(np.random.default_rng(n), False, n, n) + 4 * np.eye(n)
    with Device(gpu_lib) as d:
        p = [d.put(a), d.put(np.zeros(n, np.int64)), d.put(np.zeros(n, np.int32)), d.put(np.zeros((n, n)))]
        assert gpu_lib.peec_gb300_lu_factor_device(p[0], n, 1e-14, p[1], p[2], None, None) == 0
        assert gpu_lib.peec_gb300_inverse_device(p[0], p[2], n, p[3]) == 0
        lu, perm, x = d.get(p[0], a), d.get(p[2], np.zeros(n, np.int32)), d.get(p[3], a)
    l, u = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    cols = sorted({0, 1, 31, 32, 63, 64, 255, 256, n // 2, n - 1} & set(range(n)))
    e = abs(l @ (u @ x[:, cols]) - np.eye(n)[perm][:, cols])
    assert np.all(e <= 4 * n * U * (abs(l) @ (abs(u) @ abs(x[:, cols]))))


@pytest.mark.parametrize("nx,ny", [(21, 17), (28, 25)])
def test_transient_system_with_digits(gpu_lib, oracle, nx, ny):
    """1148 unknowns: the inverse by digit GEMMs; 2183: the factorisation too."""
    from helpers import inductance, potential
    from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh
    from test_gpu_transient import I_TOL, V_TOL, DeviceTransient, werr
    with SynthMesh.plate(0.05 * nx, 0.05 * ny, nx, ny) as m:
        _, L = inductance(gpu_lib, m)
        _, P = potential(gpu_lib, m)
        edges, R = np.ascontiguousarray(m.edges()), 1e-3 * np.ones(m.n_edges)
        src = (102900.0, 1500.0, 1.0e6, 0.0, 0, m.n_nodes - 1)
        so, Io, Vo, _ = oracle.transient_lightning(L, P, edges, R, 2, 1e-7, src, 12, probe_nodes=range(m.n_nodes),
                                                   probe_edges=range(m.n_edges))
        t = DeviceTransient(gpu_lib, L, P, edges, R, 2, 1e-7)
        try:
            s, I, V, _ = t.run(src, 12)
            assert s == 0 and so == 0
            assert werr(I, Io) < I_TOL and werr(V, Vo) < V_TOL
        finally:
            t.close()


@pytest.mark.parametrize("eps", [1e-7, 1e-10, 1e-13])
@pytest.mark.parametrize("turned", [False, True])
def test_each_part_of_complex_entries_keeps_its_own_accuracy(gpu_lib, eps, turned):
    """Imaginary parts eps of the real ones (a small resistance beside j omega L
    and the other way round: rows, inner index and columns turned by j at random):
    each part is as accurate as an FMA chain of its own products."""
    m, n, k = 150, 110, 192
    rng = np.random.default_rng(11)
    a, b, c = (rng.standard_normal(s) + 1j * eps * rng.standard_normal(s) for s in ((m, k), (k, n), (m, n)))
    if turned:
        r, s, t = (TURNS[rng.integers(0, 4, x)] for x in (m, n, k))
        a, b, c = a * r[:, None] * t[None].conj(), b * t[:, None] * s[None], c * r[:, None] * s[None]
    check(a, b, c, digit_sub(gpu_lib, a, b, c), some(m), floor=False)


@pytest.mark.parametrize("k", [1, 17, 64, 130, 192])
def test_parts_that_are_sums_of_zeros(gpu_lib, k):
    """Without the small parts (a lossless system) the other part is exactly what it was,
    and a single nonzero factor far below the rest (1e-30 or 1e-200) is not overlooked."""
    m, n = 150, 110
    rng = np.random.default_rng(12)
    r, s, t = (TURNS[rng.integers(0, 4, x)] for x in (m, n, k))
    a, b, c = (rng.standard_normal(x).astype(complex) for x in ((m, k), (k, n), (m, n)))
    a, b, c = a * r[:, None] * t[None].conj(), b * t[:, None] * s[None], c * r[:, None] * s[None]
    i = k - 1
    a[5, i] += 1e-30 * 1j * r[5] * np.conj(t[i])
    b[i, 7] += 1e-30 * 1j * t[i] * s[7]
    a[6, i] += 1e-200 * 1j * r[6] * np.conj(t[i])
    out = digit_sub(gpu_lib, a, b, c)
    check(a, b, c, out, some(m) + [5, 6], floor=False)
    small = out / r[:, None] / s[None]
    whole = np.ones((m, n), dtype=bool)
    whole[[5, 6]] = whole[:, 7] = False
    assert np.all(small.imag[whole] == 0)
    assert np.all(small.imag[[5, 6]] != 0) and np.all(small.imag[:, 7] != 0)


@pytest.mark.parametrize("eps,digits", [(0.0, 1), (1e-2, 1), (1e-9, 0)])
def test_systems_of_small_second_parts(gpu_lib, eps, digits):
    """A checked run in which FP64 FMAs would do most entries takes them from the start;
    without second parts, or with ones of the usual size, it keeps the digits."""
    n = 700
    rng = np.random.default_rng(13)
    a = rng.standard_normal((n, n)) + 1j * eps * rng.standard_normal((n, n))
    s, lu, piv, rs, cs, used = factor(gpu_lib, a, CHECKED)
    assert s == 0 and used == digits
    _, lu0, piv0, _, _, _ = factor(gpu_lib, a, FMA)
    assert np.array_equal(piv, piv0)
    if eps == 0.0:
        assert np.all(lu.imag == 0)
    if not digits:
        assert np.array_equal(lu, lu0)


@pytest.fixture
def no_digits(gpu_lib):
    """No memory for digits: their scratch is refused to this thread."""
    before = gpu_lib.peec_gb300_set_digit_scratch_limit(0)
    yield gpu_lib
    gpu_lib.peec_gb300_set_digit_scratch_limit(before)


@pytest.mark.parametrize("cplx", [False, True])
def test_factorisation_without_memory_for_digits(no_digits, cplx):
    a = normal(np.random.default_rng(14), cplx, 1400, 1400)
    want = factor(no_digits, a, FMA)
    for form in (DIGITS, CHECKED):
        got = factor(no_digits, a, form)
        assert got[0] == 0 and got[5] == 0
        assert all(np.array_equal(x, y) for x, y in zip(got[1:5], want[1:5]))


def test_host_factorisation_without_memory_for_digits(no_digits):
    from helpers import ComplexLU
    a = normal(np.random.default_rng(15), True, 1310, 1310)
    f = ComplexLU(no_digits, a)
    assert f.status == 0
    lu, piv, rs, cs = f.factors()
    f.free()
    _, lu0, piv0, rs0, cs0, _ = factor(no_digits, a, FMA)
    assert np.array_equal(lu, lu0) and np.array_equal(piv, piv0) and np.array_equal(rs, rs0) and np.array_equal(cs, cs0)


@pytest.mark.parametrize("n", [1025])
def test_inverse_without_memory_for_digits(no_digits, n):
    test_inverse(no_digits, n)


@pytest.mark.parametrize("nx,ny", [(28, 25)])
def test_transient_system_without_memory_for_digits(no_digits, oracle, nx, ny):
    test_transient_system_with_digits(no_digits, oracle, nx, ny)


def test_no_error_is_left_where_digits_are_refused(no_digits, capfd):
    capfd.readouterr()
    a = normal(np.random.default_rng(16), True, 1310, 1310)
    assert factor(no_digits, a, CHECKED)[0] == 0
    assert "ERROR" not in capfd.readouterr().err


@pytest.mark.parametrize("cplx,pivot", [(False, 1.0), (False, 1.9), (False, 0.75), (True, 1.0)])
def test_near_ties_in_late_columns(gpu_lib, cplx, pivot):
    """Two candidates of column 2112 whose rows have met no update (zeros before): a
    checked run gives the digits up where they are closer than 2^-44 + k^1.5 2^-53
    of the pivot (k = 2176, the end of the block), and twice the difference of
    2^-39 found between candidates of the two forms there is well inside."""
    first, n = 2112, 2180
    rng = np.random.default_rng(17)
    t = np.eye(n - first) + 0.1 * rng.uniform(-1, 1, (n - first,) * 2) * (1 - np.eye(n - first))
    t[1:, 0] *= 0.1
    a = np.zeros((n, n), dtype=complex if cplx else float)
    a[:first, :first] = normal(rng, cplx, first, first)
    line = 2.0 ** -44 + 2176.0 ** 1.5 * 2.0 ** -53
    for apart, digits in ((2.0 ** -38, 0), (0.8 * line, 0), (4 * line, 1)):
        t[0, 0], t[1, 0] = pivot, pivot * (1 - apart)
        a[first:, first:] = t
        s, _, piv, rs, cs, used = factor(gpu_lib, a, CHECKED)
        assert s == 0 and piv[first] == first and used == digits
        assert not cplx or (np.all(rs[first:] == 1) and np.all(cs[first:] == 1))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("form", [DIGITS, CHECKED])
def test_status_of_systems_that_are_singular_to_rounding(gpu_lib, cplx, form):
    """The last column a combination of others: the last pivot is rounding, another
    one by digits than by FP64 FMAs, and for every tolerance around it FP64 FMAs
    say whether the matrix is refused."""
    n, refused = 200, 0
    for seed in range(4):
        rng = np.random.default_rng(seed)
        a = normal(rng, cplx, n, n)
        a[:, -1] = a[:, :-1] @ (rng.integers(-3, 4, n - 1) / 16.0)
        for tol in 2.0 ** np.arange(-62.0, -46.0, 0.5):
            want = factor(gpu_lib, a, FMA, tol)[0]
            refused += want != 0
            assert factor(gpu_lib, a, form, tol)[0] == want
    assert 0 < refused < 4 * 32


def test_inverse_outside_the_middle_of_the_range(gpu_lib):
    """Quotients whose divisor's reciprocal overflows, or whose dividend is infinite,
    are those of a division."""
    for u, want in ((np.array([[1e-310, 1e-10], [0.0, 1.0]]), [[np.inf, -1e-10 / 1e-310], [0.0, 1.0]]),
                    (np.array([[2.0, np.inf], [0.0, 1.0]]), [[np.nan, -np.inf], [0.0, 1.0]]),  # 1 - inf 0
                    (np.array([[1e300, 1e-20], [0.0, 1e-5]]), [[1e-300, -1e-20 * 1e5 / 1e300], [0.0, 1e5]])):
        with Device(gpu_lib) as d:
            p = [d.put(u), d.put(np.arange(2, dtype=np.int32)), d.put(np.zeros((2, 2)))]
            assert gpu_lib.peec_gb300_inverse_device(p[0], p[1], 2, p[2]) == 0
            assert np.allclose(d.get(p[2], u), want, rtol=4 * U, atol=5e-324, equal_nan=True)
