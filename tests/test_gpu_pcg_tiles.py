"""texo_gp_quadratic_solve where its layout of the matrix can go wrong: rows of
a segment (16 entries) less or more one, empty rows, one row, systems of a
tile (512 segments) less or more one, more tiles than multiprocessors, and a
row longer than 512 segments, which is a tile by itself with longer ones.

The systems are diagonally dominant (condition about 4), so the residuals'
rounding is below 1e-15 of |b| and a residual of 1e-4 |r0| is known to 1e-11:
its square is held to 1e-8. With the oracle's iteration count the iterates
agree to rounding, here to 1e-10 of the largest."""
import numpy as np
import pytest

from oracle import ffi
from texo_gb300.placer import quadratic_solve


def ring_system(n, degrees, hub, seed_no):
    rng = np.random.default_rng(seed_no)
    a, b = [], []
    for k in range(1, max(degrees) // 2 + 2):   # row i reaches 2 (k - 1) neighbours or more where its degree asks for it
        i = np.arange(n)[np.resize(degrees, n) >= 2 * k]
        j = (i + k) % n
        a.append(i[j != i])
        b.append(j[j != i])
    if hub:
        others = np.arange(1, n)
        a.append(np.zeros(n - 1, np.int64))
        b.append(others)
    a, b = np.concatenate(a), np.concatenate(b)
    w = rng.uniform(0.1, 1.0, a.size)
    rows, cols, ww = np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w])
    order = np.argsort(rows, kind="stable")
    ptr = np.zeros(n + 1, np.int64)
    np.add.at(ptr, rows + 1, 1)
    diag = np.zeros(n)
    np.add.at(diag, rows, ww)
    return 1.7 * diag + 0.5, np.cumsum(ptr), cols[order], ww[order], rng.normal(size=n), rng.normal(size=n)


@pytest.mark.gpu
@pytest.mark.parametrize("n,degrees,hub", [
    (1, [0], False), (33, [0, 2], False), (511, [14, 16, 18], False), (513, [30, 32, 34, 0], False),
    (4000, [16], False), (20000, [0, 2, 14, 18, 66], False), (9000, [4], True), (100000, [12, 20], False)])
def test_the_dealt_matrix_solves_as_the_rows_do(n, degrees, hub):
    diag, ptr, idx, w, rhs, x0 = ring_system(n, degrees, hub, n)
    xr, sr, ok = ffi.solve_quadratic(diag, ptr, idx, w, rhs, x0)
    xg, sg = quadratic_solve(diag, ptr, idx, w, rhs, x0)
    assert ok and sg["stop"] == "residual"
    assert abs(sg["iterations"] - sr.iterations) <= 2
    assert abs(sg["initial_residual_squared"] - sr.initial_residual_squared) <= 1e-12 * sr.initial_residual_squared
    rows = np.repeat(np.arange(n), np.diff(ptr))
    res = rhs - diag * xg + np.bincount(rows, w * xg[idx], minlength=n)
    assert abs(float(res @ res) - sg["final_residual_squared"]) <= 1e-8 * sg["target_squared"]
    if sg["iterations"] == sr.iterations:
        assert np.max(np.abs(xg - xr)) <= 1e-10 * np.max(np.abs(xr))
