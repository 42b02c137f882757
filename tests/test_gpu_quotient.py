"""The quadratic solve's division by the diagonal against IEEE division.

Before its last rounding the corrected quotient is within 1.5 * 2^-53 units in
the last place (ulp) of a / b: random operands meet a tie that close with a
probability of 2^-51, so a million give the rounded quotient exactly. Quotients
placed next to ties, significands of all ones and powers of two may differ by
one ulp, numerators and quotients at the subnormal end by one spacing there.
Diagonals that have no reciprocal are divided by, exactly; a solve with such
ones takes the oracle's iterations to its answer, to 1e-10 as the other solves."""
import ctypes as C

import numpy as np
import pytest

from oracle import ffi
from texo_gb300 import abi
from texo_gb300.placer import quadratic_solve

pytestmark = pytest.mark.gpu
N = 1 << 20


def quotient(a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    out = np.empty_like(a)
    lib = abi.load()
    abi.check(lib.texo_gp_selftest_quotient(0, a.size, abi.ptr(a, C.c_double), abi.ptr(b, C.c_double),
                                            abi.ptr(out, C.c_double)), "texo_gp_selftest_quotient")
    return out


def significands(rng, n):
    return 1.0 + rng.integers(0, 1 << 52, n) * 2.0**-52


def test_random_operands_give_the_rounded_quotient():
    rng = np.random.default_rng(1)
    for span in (0, 30, 300):
        a = significands(rng, N) * 2.0 ** rng.integers(-span, span + 1, N) * rng.choice([-1.0, 1.0], N)
        b = significands(rng, N) * 2.0 ** rng.integers(-min(span, 600), min(span, 600) + 1, N)
        assert np.array_equal(quotient(a, b), a / b)


def test_quotients_next_to_ties_and_extreme_significands():
    rng = np.random.default_rng(2)
    b = significands(rng, N)
    ones = 2.0 - 2.0**-52
    b[: N // 4] = ones
    b[N // 4: N // 2] = 2.0 ** rng.integers(-600, 601, N // 4)
    middle = significands(rng, N) * (1 + 2.0**-53)
    a = b * middle
    a[::3] = np.nextafter(a[::3], np.inf)
    a[::7] = ones
    exact = a / b
    assert np.all(np.abs(quotient(a, b) - exact) <= np.spacing(np.abs(exact)))


@pytest.mark.parametrize("ea,eb", [((-1074, -1000), (-600, 600)), ((-1074, -1060), (-1, 1)), ((-700, -600), (350, 600))])
def test_the_subnormal_end(ea, eb):
    rng = np.random.default_rng(3)
    a = np.ldexp(significands(rng, N), rng.integers(ea[0], ea[1], N))
    b = np.ldexp(significands(rng, N), rng.integers(eb[0], eb[1], N))
    b = np.clip(b, 1e-199, 1e199)
    with np.errstate(under="ignore"):
        exact = a / b
    assert np.all(np.abs(quotient(a, b) - exact) <= np.spacing(np.abs(exact)))


def test_diagonals_without_a_reciprocal_are_divided_by():
    rng = np.random.default_rng(4)
    b = np.concatenate([np.ldexp(significands(rng, 1000), rng.integers(-1022, -680, 1000)),
                        np.ldexp(significands(rng, 1000), rng.integers(680, 1023, 1000)), [1e-200, 1e200]])
    with np.errstate(under="ignore", over="ignore"):
        for scale in (1e-30, 1.0, 1e30):
            a = significands(rng, b.size) * scale
            assert np.array_equal(quotient(a, b), a / b)


def test_a_solve_with_such_diagonals_is_the_oracles():
    n = 200
    rng = np.random.default_rng(5)
    ptr = np.concatenate([2 * np.arange(n + 1), np.full(80, 2 * n)])
    i = np.arange(n)
    idx = np.stack([(i + 1) % n, (i - 1) % n], axis=1).reshape(-1)
    diag = np.concatenate([rng.uniform(2.5, 4.0, n), np.full(40, 3e-205), np.full(40, 7e201)])
    rhs = np.concatenate([rng.normal(size=n), 1e-204 * rng.uniform(1, 2, 40), rng.normal(size=40)])
    x0 = np.zeros(n + 80)
    xr, sr, ok = ffi.solve_quadratic(diag, ptr, idx, np.ones(2 * n), rhs, x0)
    x, s = quadratic_solve(diag, ptr, idx, np.ones(2 * n), rhs, x0)
    assert ok and s["stop"] == "residual" and s["iterations"] == sr.iterations > 2
    for part in (slice(0, n), slice(n, n + 40), slice(n + 40, n + 80)):
        assert np.max(np.abs(x[part] - xr[part])) <= 1e-10 * np.max(np.abs(xr[part]))
