"""The FP32 fitter's solve and gain-ratio decisions, piece by piece: the fp32
gain test decides exactly as FP64 wherever it decides; the solve equals an FP64
restatement on definite, indefinite, degenerate and badly scaled systems."""
import ctypes

import numpy as np
import pytest
import torch

from pycompute_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _t(a, dt=None):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _solve(P, A, b, s, f, ftp, mu=0.25, eta=0.75):
    n = b.shape[1]
    args = [_t(v.astype(np.float32)) for v in (A, b, s, f, ftp)]
    x = torch.empty((P, n), device=DEV)
    code = torch.empty(n, dtype=torch.int32, device=DEV)
    _lib.check("pcgb_solve_helpers", _lib.lib().pcgb_solve_helpers(
        P, *[_ptr(a) for a in args], mu, eta, _ptr(x), _ptr(code), n,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return x.cpu().numpy(), code.cpu().numpy()


def _gmw64(A, b, out=np.float32):
    """The GMW81 solve (solver.py:23-95, 431-463): scaling in A's type, the rest in double, one system per column."""
    P, n = b.shape
    rot = [P - 1] + list(range(P - 1))
    at = lambda i, j: A[max(i, j) * (max(i, j) + 1) // 2 + min(i, j)]  # noqa: E731
    with np.errstate(all="ignore"):
        s = [np.sqrt(np.abs(at(rot[i], rot[i]))) for i in range(P)]
        L = [[(at(rot[i], rot[j]) / (s[i] * s[j])).astype(np.float64) for j in range(i + 1)] for i in range(P)]
        y = [(b[rot[i]] / s[i]).astype(np.float64) for i in range(P)]
        mx = lambda m, v: np.where(v > m, v, m)  # noqa: E731 - a NaN never wins
        gam, nu = np.zeros(n), np.zeros(n)
        for i in range(P):
            gam = mx(gam, np.abs(L[i][i]))
            for j in range(i):
                nu = mx(nu, np.abs(L[i][j]))
        nu = nu / np.sqrt(P * P - 1.0)
        beta2 = mx(mx(np.full(n, 4e-16), gam), nu)
        delta = np.where(gam + nu > 1, 4e-16 * (gam + nu), 4e-16)
        d = []
        for j in range(P):
            Lj = [L[j][q] / d[q] for q in range(j)]
            th = np.zeros(n)
            for i in range(j + 1, P):
                for q in range(j):
                    L[i][j] = L[i][j] - Lj[q] * L[i][q]
                th = mx(th, np.abs(L[i][j]))
            L[j][:j] = Lj
            dj = np.abs(L[j][j])
            dj = np.where(dj < delta, delta, dj)
            dj = np.where(dj < th * th / beta2, th * th / beta2, dj)
            d.append(dj)
            for i in range(j + 1, P):
                L[i][i] = L[i][i] - L[i][j] ** 2 / dj
        for i in range(P):
            for j in range(i):
                y[i] = y[i] - L[i][j] * d[j] * y[j]
            y[i] = y[i] / d[i]
        for i in reversed(range(P)):
            for j in range(i + 1, P):
                y[i] = y[i] - L[j][i] * y[j]
        x = [None] * P
        for i in range(P):
            x[rot[i]] = (y[i] * (A.dtype.type(1) / s[i]).astype(np.float64)).astype(out)
    return np.stack(x)


def _systems(P, n, kind, rng):
    J = rng.standard_normal((P + 2, P, n))
    A = np.einsum("kin,kjn->ijn", J, J)
    for i in range(P):
        A[i, i] += 0.3
        if kind == "indefinite":
            A[i, i] -= rng.uniform(0.0, 2.0 * P, n)
    scale = {"wide": 30, "huge": 55}.get(kind, 3)
    e = 2.0 ** rng.integers(-scale, scale + 1, (P, n))
    A, b = A * e[:, None] * e[None], rng.standard_normal((P, n)) * e
    if kind == "zeros":
        for i in range(P):
            for j in range(i):
                z = rng.random(n) < 0.5
                A[i, j][z] = A[j, i][z] = 0.0
            b[i][rng.random(n) < 0.3] = 0.0
    A, b = A.astype(np.float32), b.astype(np.float32)
    if kind == "nan":
        b[0, ::3] = np.nan
        A[0, 0, 1::3] = np.inf
        A[P - 1, 0, 2::3] = A[0, P - 1, 2::3] = np.nan
    return np.stack([A[i, j] for i in range(P) for j in range(i + 1)]), b


@pytest.mark.parametrize("P", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("kind", ["definite", "indefinite", "wide", "huge", "zeros", "nan"])
def test_solve_equals_fp64_restatement(P, kind):
    n = 4099
    A, b = _systems(P, n, kind, np.random.default_rng(P))
    z = np.zeros(n)
    x, _ = _solve(P, A, b, np.zeros((P, n)), z, z)
    ref = _gmw64(A, b)
    fine = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(x), fine)
    # one float rounding of a solve that is exact to 2^-52 times the pivots' growth (|c| / d <= 1e4 for all but a few
    # of these random systems); small entries carry the error of the largest scaled one
    size = np.abs(np.where(fine, ref, 0)) * np.sqrt(np.abs(np.stack([A[i * (i + 1) // 2 + i] for i in range(P)])))
    with np.errstate(all="ignore"):
        tol = 2.0 ** -23 * np.abs(ref) + 1e-10 * size.max(0) / np.sqrt(
            np.abs(np.stack([A[i * (i + 1) // 2 + i] for i in range(P)]))) + 1.5e-45
        bad = fine & (np.abs(x - ref) > tol)
    assert bad.mean() < 1e-3, bad.mean()


@pytest.mark.parametrize("P", [2, 4, 6])
@pytest.mark.parametrize("mu,eta", [(0.25, 0.75), (0.0, 0.75), (-0.5, 2.0)])
def test_fp32_gain_decides_as_fp64(P, mu, eta):
    rng = np.random.default_rng(17 + P)
    n = 1 << 18
    A, b = _systems(P, n, "definite", rng)
    s = rng.standard_normal((P, n)) * 2.0 ** rng.integers(-24, 3, n) / np.sqrt(
        np.stack([A[i * (i + 1) // 2 + i] for i in range(P)]))
    s32 = s.astype(np.float32).astype(np.float64)
    pred = np.zeros(n)
    for i in range(P):
        pred += s32[i] * b[i]
        for j in range(i + 1):
            pred -= A[i * (i + 1) // 2 + j].astype(np.float64) * s32[i] * s32[j] * (0.5 if i == j else 1.0)
    # actual reductions around both thresholds (some exactly on the rounded threshold), ties, noise and non-finite costs
    f = rng.uniform(0.0, 1.0, n) * np.abs(pred) * 8
    k = rng.integers(0, 8, n)
    ftp = f - np.select([k == 0, k == 1, k == 2, k == 3], [2 * mu * pred * (1 + rng.normal(0, 1e-6, n)),
                                                             2 * eta * pred * (1 + rng.normal(0, 1e-6, n)),
                                                             np.zeros(n), 2 * eta * pred], rng.normal(0, 2, n) * pred)
    ftp[::97], f[1::97], s[:, 2::97] = np.nan, np.inf, 0.0
    _, code = _solve(P, A, b, s, f, ftp, mu, eta)
    told = (code & 8) != 0
    np.testing.assert_array_equal((code & 7)[told], (code >> 4)[told])
    regular = (np.arange(n) % 97 > 2) & (k > 3)
    assert told[regular].mean() > 0.97


def _scalars(a, b, x):
    n = len(a)
    ta, tb, tx = _t(a), _t(b), _t(x)
    root, quot, prod = (torch.empty(n, device=DEV) for _ in range(3))
    rcp = torch.empty(n, dtype=torch.float64, device=DEV)
    ok = torch.zeros(n, dtype=torch.int32, device=DEV)
    _lib.check("pcgb_scalar_helpers", _lib.lib().pcgb_scalar_helpers(
        _ptr(ta), _ptr(tb), _ptr(tx), _ptr(root), _ptr(quot), _ptr(rcp), _ptr(prod), _ptr(ok), n,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return [v.cpu().numpy() for v in (root, quot, rcp, prod, ok)]


def test_straight_line_root_and_quotient_are_correctly_rounded():
    mant = np.arange(1 << 23, dtype=np.uint32)
    rng = np.random.default_rng(5)
    for e in (127, 128, 77, 190):  # every significand, both exponent parities
        b = (mant | np.uint32(e << 23)).view(np.float32)
        a = (rng.integers(0, 1 << 23, len(b)).astype(np.uint32) | np.uint32(120 << 23)).view(np.float32)
        a[::3] = np.nextafter(b[::3], np.float32(0)) * np.float32(0.5)
        root, quot, *_ = _scalars(a, b, np.ones(len(b)))
        np.testing.assert_array_equal(root, np.sqrt(b))
        np.testing.assert_array_equal(quot, a / b)


def test_integer_reciprocal_and_fp32_product_equal_the_fp64_ones():
    rng = np.random.default_rng(6)
    n = 1 << 22
    m = rng.uniform(1.0, 2.0, n)
    m[::5] = 1.0 + rng.integers(0, 1 << 12, len(m[::5])) * 2.0 ** -52   # a seed that starts at a power of two
    m[1::5] = 2.0 - rng.integers(1, 1 << 12, len(m[1::5])) * 2.0 ** -52
    m[2::5] = m[2::5].astype(np.float32)
    x = np.ldexp(m, rng.integers(-130, 130, n))
    a = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-40, 40, n)).astype(np.float32)
    x = np.where(np.arange(n) % 11 == 0, -x, x)
    x[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e300, 1e-300]
    _, _, rcp, prod, ok = _scalars(a, np.ones(n, np.float32), x)
    want = torch.empty(n, dtype=torch.float64, device=DEV)
    tx = _t(x)
    _lib.check("pcgb_fp64_helpers", _lib.lib().pcgb_fp64_helpers(_ptr(tx), _ptr(want), None, n, ctypes.c_void_p(
        torch.cuda.current_stream().cuda_stream)))
    told = (ok & 1) != 0
    np.testing.assert_array_equal(rcp.view(np.int64)[told], want.cpu().numpy().view(np.int64)[told])
    assert not told[:8].any() and not told[x < 0].any()
    mid = (np.abs(np.log2(np.abs(np.where(x == 0, 1, x)))) < 100) & (x > 0)
    assert told[mid].mean() > 0.99
    with np.errstate(all="ignore"):
        both = (x * a.astype(np.float64)).astype(np.float32)
    told = (ok & 2) != 0
    np.testing.assert_array_equal(prod.view(np.int32)[told], both.view(np.int32)[told])
    near = np.abs(np.log2(np.abs(np.where(x == 0, 1, x)))) < 25
    assert told[near & np.isfinite(x) & (x != 0)].mean() > 0.99 and not told[:8].any()


@pytest.mark.parametrize("P", [2, 4, 6])
@pytest.mark.parametrize("kind", ["definite", "indefinite", "zeros", "nan"])
def test_double_solver_keeps_the_rules_of_its_maxima(P, kind):
    """The all-double solve, whose maxima run on bit patterns, against the numpy rules (a NaN never wins)."""
    from pycompute_gb300 import GMW81Solver

    n = 1027
    A, b = (v.astype(np.float64) for v in _systems(P, n, kind, np.random.default_rng(P + 50)))
    x = torch.empty((P, n), dtype=torch.float64, device=DEV)
    GMW81Solver(P, torch.float64).run(_t(A), _t(b), None, x)
    got = x.cpu().numpy()
    ref = _gmw64(A, b, np.float64)
    fine = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(got), fine)
    d = np.sqrt(np.abs(np.stack([A[i * (i + 1) // 2 + i] for i in range(P)])))
    with np.errstate(all="ignore"):
        # rounding (2^-53) times the pivots' growth, as for the float solve above
        bad = fine & (np.abs(got - ref) > 1e-9 * (np.abs(np.where(fine, ref, 0)) * d).max(0) / d + 1e-300)
    assert bad.mean() < 1e-3, bad.mean()


@pytest.mark.parametrize("P", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_a_diagonal_that_is_not_finite_leaves_no_unknown(P, value):
    """One such entry at every position, beside entries of every kind: no unknown is finite, as in the restatement."""
    rng = np.random.default_rng(P + 90)
    for kind in ("definite", "indefinite", "zeros"):
        for i in range(P):
            A, b = (v.copy() for v in _systems(P, 257, kind, rng))
            A[i * (i + 1) // 2 + i] = value
            x, _ = _solve(P, A, b, np.zeros_like(b), np.ones(257), np.ones(257))
            assert not np.isfinite(_gmw64(A, b)).any()
            assert not np.isfinite(x).any()
