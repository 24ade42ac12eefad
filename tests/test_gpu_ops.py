"""The arithmetic headers' own reciprocals, quotients and roots on the device,
operation by operation, against the compiler's (tests/ops_check.cu, built here
with the library's flags)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
INF, NAN = np.inf, np.nan


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    """ops(flavour, name, rows, nout): result rows of one operation."""
    from tests.conftest import gpu_available
    if not gpu_available():
        pytest.skip("no CUDA device")
    from cfd_inwsl_b200 import build_ext
    try:
        nvcc = build_ext.nvcc_path()
    except RuntimeError:
        pytest.skip("no nvcc")
    libs = {}

    def call(flavour, name, rows, nout):
        if flavour not in libs:
            out = tmp_path_factory.mktemp("ops") / f"ops_{flavour}.so"
            flags = ["--fmad=false"] if flavour == "strict" else ["--fmad=true", "-DCFD_FAST"]
            subprocess.run([nvcc] + build_ext.common_flags() + flags + ["-shared", str(ROOT / "tests" / "ops_check.cu"),
                                                                        "-o", str(out)], check=True)
            libs[flavour] = C.CDLL(str(out))
        x = np.ascontiguousarray(rows, dtype=np.float64)
        r = np.empty((len(x), nout))
        f = getattr(libs[flavour], "ops_" + name)
        f.argtypes = [C.c_void_p, C.c_void_p, C.c_long]
        assert f(x.ctypes.data, r.ctypes.data, len(x)) == 0
        return r

    return call


def normals(rng, n, lo, hi):
    """Positive numbers with exponents lo .. hi - 1, significands random and
    next to the ends of a binade."""
    m = 1 + rng.random(n)
    k = rng.random(n)
    ulps = rng.integers(0, 16, n)
    m = np.where(k < 0.2, 2 - (1 + ulps) * 2.0**-52, m)
    m = np.where(k > 0.8, 1 + ulps * 2.0**-52, m)
    return np.ldexp(m, rng.integers(lo, hi, n))


def spec_operands():
    """Dividends and divisors in range with exponents from end to end, the
    all-ones significand and its neighbours at every exponent, zeros."""
    rng = np.random.default_rng(0)
    n = 1 << 20
    b = normals(rng, n, -400, 200)
    a = normals(rng, n, -800, 500) * rng.choice([-1.0, 1.0], n)
    e = np.arange(-400, 200)
    edge = np.concatenate([np.ldexp(2 - k * 2.0**-52, e) for k in (1, 2, 3)] + [np.ldexp(1 + k * 2.0**-52, e) for k in (0, 1, 2)])
    ends_a = np.ldexp(rng.uniform(1, 2, 64), np.resize([-800, -799, 498, 499], 64))
    b = np.concatenate([b, edge, edge, np.repeat(edge, 64)])
    a = np.concatenate([a, np.zeros(len(edge)), -np.zeros(len(edge)), np.tile(ends_a, len(edge))])
    return np.stack([a, b], 1)


def test_branch_free_operations_strict(ops):
    """Taken for every operand in range and rounded as the compiler's."""
    x = spec_operands()
    r = ops("strict", "spec", x, 9)
    assert (r[:, [1, 4, 7]] == 1).all()
    for k in (0, 3, 6):
        np.testing.assert_array_equal(r[:, k].view(np.uint64), r[:, k + 2].view(np.uint64))


def test_branch_free_operations_fast(ops):
    """The same operations in the fast flavour: quotients and roots keep their
    correction; its reciprocal is the cubic step alone, within an ulp, and its
    reciprocal root within 1.5 roundings of 2^-53 (the residual's product and
    the result's) and the step's own error."""
    x = spec_operands()
    r = ops("fast", "spec", x, 9)
    assert (r[:, [1, 4, 7]] == 1).all()
    for k in (0, 3, 6):
        assert (np.abs(r[:, k] - r[:, k + 2]) <= np.spacing(np.abs(r[:, k + 2]))).all()
    b = x[:, 1]
    r = ops("fast", "rsqrt", b[:, None], 2)
    assert (r[:, 1] == 1).all()
    want = 1 / np.sqrt(b.astype(np.longdouble))
    assert (np.abs(r[:, 0] - want) <= (1.5 * 2.0**-53 + 2.0**-56) * want).all()


@pytest.mark.parametrize("flavour", ["strict", "fast"])
def test_branch_free_operations_leave_other_operands(ops, flavour):
    """Operands outside the ranges, next to their ends among them, are refused:
    the callers evaluate those out of line."""
    below, above = np.nextafter(2.0**-400, 0), 2.0**200
    for v in (below, 2.0**-401, above, 2.0**201, 0.0, -0.0, -1.0, INF, NAN, 5e-324):
        r = ops(flavour, "spec", [[1.0, v]], 9)[0]
        assert (r[[1, 4, 7]] == 0).all(), v
    for v in (np.nextafter(2.0**-800, 0), 5e-324, -(2.0**-801), 2.0**500, -(2.0**501), INF, NAN):
        assert ops(flavour, "spec", [[v, 1.0]], 9)[0, 1] == 0, v


def test_division_by_a_sum_of_weights(ops):
    """WENO-Z's last division: taken and rounded as the compiler's while the
    quotient is 0 or within 2^-960 .. 2^1000, refused next to and beyond the
    ends (a refused one is only computed again)."""
    rng = np.random.default_rng(7)
    b = normals(rng, 1 << 20, 0, 1000)
    q = normals(rng, 1 << 20, -959, 20) * rng.choice([-1.0, 1.0], 1 << 20)
    q[:1000], q[1000:2000] = 0.0, -0.0
    edge = np.concatenate([np.ldexp(2 - k * 2.0**-52, np.arange(1000)) for k in (1, 2)] + [np.ldexp(1.0, np.arange(1000))])
    b = np.concatenate([b, edge])
    a = np.concatenate([q, rng.normal(size=len(edge))]) * b
    r = ops("strict", "div_sum", np.stack([a, b], 1), 3)
    assert (r[:, 1] == 1).all()
    np.testing.assert_array_equal(r[:, 0].view(np.uint64), r[:, 2].view(np.uint64))
    bad = [[1.0, 2.0**1000], [1.0, INF], [1.0, NAN], [NAN, 1.0], [INF, 1.0], [1e-300, 2.0**600], [2.0**1010, 1.0]]
    assert (ops("strict", "div_sum", bad, 3)[:, 1] == 0).all()


@pytest.mark.parametrize("flavour", ["strict", "fast"])
def test_wenoz_beside_a_flat_side(ops, flavour):
    """Stencils of equal values, with a jump or noise beside them: a weight
    there is the square of the jump's measure over 1e-40 and was refused, so
    that the whole face was computed twice. Taken, and equal to the compiler's
    operations (strict) or within the spread's rounding (fast: its quotients
    are the same, sums are contracted)."""
    rng = np.random.default_rng(8)
    q = np.ones((20000, 5)) * rng.normal(size=(20000, 1))
    jump = rng.integers(1, 5, len(q))
    size = rng.normal(size=(len(q), 1)) * 10.0**rng.integers(-12, 9, (len(q), 1))
    q += (np.arange(5) >= jump[:, None]) * size
    q[::3] += 1e-15 * rng.normal(size=(len(q[::3]), 5))
    r = ops(flavour, "wenoz", q, 3)
    assert (r[:, 1] == 1).all()
    if flavour == "strict":
        np.testing.assert_array_equal(r[:, 0].view(np.uint64), r[:, 2].view(np.uint64))
    else:
        # two evaluations of one formula: candidates within 8 roundings of the
        # stencil's largest value each, weights positive
        assert (np.abs(r[:, 0] - r[:, 2]) <= 16 * 2.0**-52 * np.abs(q).max(1)).all()


def test_adjoint_reciprocal_and_root(ops):
    """Within an ulp of the compiler's for normal operands: a cubic step from a
    seed off by less than 2^-18 leaves 2^-54, and one rounding half an ulp."""
    rng = np.random.default_rng(1)
    b = normals(rng, 1 << 20, -1022, 1022) * rng.choice([-1.0, 1.0], 1 << 20)
    got, want = ops("fast", "arcp", b[:, None], 2).T
    assert (np.abs(got - want) <= np.spacing(np.abs(want))).all()
    x = normals(rng, 1 << 20, -900, 1022)
    got, want = ops("fast", "asqrt", x[:, None], 2).T
    assert (np.abs(got - want) <= np.spacing(want)).all()


def test_adjoint_of_an_overflowed_measure(ops):
    """A stencil whose outer value overflows a smoothness measure: its weight is
    0, and the gradient is that of the candidates left, finite and with a sum
    of 1 (each candidate reproduces a constant)."""
    rng = np.random.default_rng(2)
    rows = []
    for big in (1e155, -1e160, 1e200):
        for at in (0, 4):
            q = rng.normal(size=5) * 1e-3
            q[at] = big
            rows.append([*q, 1.0])
    g = ops("fast", "wcns5_adj", rows, 5)
    assert np.isfinite(g).all()
    # the measures' own derivatives sum to rounding: beta does not see a constant
    np.testing.assert_allclose(g.sum(1), 1.0, rtol=0, atol=1e-9)


def left_density(U):
    """Density of the left face state of six cells' cons along x (WCNS5)."""
    def prim(c):
        u, v = c[1] / c[0], c[2] / c[0]
        p = 0.4 * (c[3] - 0.5 * c[0] * (u * u + v * v))
        return np.sqrt(c[0]), u, v, 0.5 * (u * u + v * v) + 3.5 * p / c[0]
    (s1, u1, v1, H1), (s2, u2, v2, H2) = prim(U[2]), prim(U[3])
    u, v, H = ((s1 * a + s2 * b) / (s1 + s2) for a, b in ((u1, u2), (v1, v2), (H1, H2)))
    ek = 0.5 * (u * u + v * v)
    h = H - ek
    c = np.sqrt(0.4 * h)
    rows = [[h - ek, u, v, -1.0], [0.5 * (u / c + ek / h), 0.5 * (-1 / c - u / h), -0.5 * v / h, 0.5 / h],
            [0.5 * (-u / c + ek / h), 0.5 * (1 / c - u / h), -0.5 * v / h, 0.5 / h]]
    Q = []
    for L in rows:
        q = U[:5] @ np.array(L)
        s = [1e-6 + (q[0] - 2 * q[1] + q[2])**2 + 0.25 * (q[0] - 4 * q[1] + 3 * q[2])**2,
             1e-6 + (q[1] - 2 * q[2] + q[3])**2 + 0.25 * (q[1] - q[3])**2,
             1e-6 + (q[2] - 2 * q[3] + q[4])**2 + 0.25 * (3 * q[2] - 4 * q[3] + q[4])**2]
        w = np.array([1 / 16, 5 / 8, 5 / 16]) / np.square(s)
        cand = [0.375 * q[0] - 1.25 * q[1] + 1.875 * q[2], -0.125 * q[1] + 0.75 * q[2] + 0.375 * q[3],
                0.375 * q[2] + 0.75 * q[3] - 0.125 * q[4]]
        Q.append(w @ cand / w.sum())
    return Q[0] / h + Q[1] + Q[2]


def test_face_density_that_cancels(ops):
    """Faces whose left density lies within a few roundings of zero, zero
    itself among them: its pressure is then -inf, which takes the positivity
    fallback, so every gradient is finite. Small amplitudes keep the weights
    linear, so that a high second cell pulls the interpolated density down to
    zero."""
    rng = np.random.default_rng(3)
    rows = []
    for _ in range(200):
        u, v = rng.uniform(0.2, 0.6, (2, 6))

        def cells(t):
            rho = 1e-3 * np.array([1.0, t, 0.1, 0.1, 1.0, 1.0])
            return np.stack([rho, rho * u, rho * v, 1e-3 / 0.4 + 0.5 * rho * (u * u + v * v)], -1)

        lo, hi = 0.1, 1.0
        assert left_density(cells(lo)) > 0 > left_density(cells(hi))
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if left_density(cells(mid)) > 0 else (lo, mid)
        for k in range(-40, 41):
            rows.append([*cells(lo + k * np.spacing(lo)).ravel(), *rng.normal(size=4)])
    assert np.isfinite(ops("fast", "face_vjp", rows, 24)).all()


def wcns5(q):
    """weno5_JSchen in extended precision, one row of five values a result."""
    q = q.astype(np.longdouble).T
    s = [(q[0] - 2 * q[1] + q[2])**2 + (q[0] - 4 * q[1] + 3 * q[2])**2 / 4,
         (q[1] - 2 * q[2] + q[3])**2 + (q[1] - q[3])**2 / 4,
         (q[2] - 2 * q[3] + q[4])**2 + (3 * q[2] - 4 * q[3] + q[4])**2 / 4]
    w = [g / (np.longdouble(1e-6) + b)**2 for g, b in zip((1 / 16, 5 / 8, 5 / 16), s)]
    u = [0.375 * q[0] - 1.25 * q[1] + 1.875 * q[2], -0.125 * q[1] + 0.75 * q[2] + 0.375 * q[3],
         0.375 * q[2] + 0.75 * q[3] - 0.125 * q[4]]
    return sum(a * b for a, b in zip(w, u)) / sum(w)


@pytest.mark.parametrize("amplitude", [1e-6, 1e-2, 1.0, 1e4, 1e7, 1e9, 1e12, 1e25])
def test_fast_wcns5_pair(ops, amplitude):
    """Both states of a face from shared differences, for differences from the
    smallest to shocks in SI units: taken by the branch-free path and within
    rounding of extended precision. A weight's relative error is below 64
    roundings (its measure's, squared, times another), which moves the mean of
    candidates by as many roundings of twice their spread of ten differences."""
    rng = np.random.default_rng(6)
    q = rng.normal(size=(20000, 6)) * amplitude
    jump = rng.integers(1, 6, len(q))
    q += (np.arange(6) >= jump[:, None]) * amplitude * 10
    q[::4] = np.where(np.arange(6) >= jump[::4, None], amplitude, 0.0)  # one clean jump
    r = ops("fast", "wcns5_pair", q, 3)
    assert (r[:, 2] == 1).all()
    spread = np.abs(np.diff(q, axis=1)).max(1)
    tol = 64 * 2 * 10 * 2.0**-53 * spread + 2.0**-52 * np.abs(q).max(1)
    assert (np.abs(r[:, 0] - wcns5(q[:, :5])) <= tol).all()
    assert (np.abs(r[:, 1] - wcns5(q[:, :0:-1])) <= tol).all()


def test_fast_wcns5_pair_leaves_what_it_does_not_cover(ops):
    """Differences whose measures leave the range, infinities and NaN."""
    q = np.zeros((5, 6))
    q[:, 3:] = np.array([1e40, 1e80, 1e160, INF, NAN])[:, None]
    assert (ops("fast", "wcns5_pair", q, 3)[:, 2] == 0).all()
