"""The kernels at the sizes where their tiles, groups and shared-memory copies
end.

- transforms of every length from 2 to 1024, square and not, alone, several
  vectors to a group and fewer than a group holds: potential against the FP64 oracle, 1e-6 normwise as for
  the other grids of this form (double-float butterflies, the FP32 storage
  between the passes decides).
- the placement loop with objects beyond the ones a block keeps in shared
  memory (1536 a block) and tile maps beyond 512, with few and many groups, and
  with every object stacked on one point: a job in a batch, whose blocks keep
  nothing and share the work otherwise, gives the targets bit for bit.
- deposits of 1 to 32 lanes on one bin, with charges on both sides of 2^17:
  the fixed-point grids are the oracle's, bit for bit.
- coordinates that are not finite are refused and the outputs left alone.
- the register clustering's window around the ends of its table's intervals
  and of its reach, a pair a control set (so that warps meet several): areas to
  1e-12, as the other cases (window values to 1e-15, sums of a few)."""
import ctypes as C

import numpy as np
import pytest

from oracle import ffi
from texo_gb300 import abi, problem as P, routability
from texo_gb300.placer import Batch, Placer, default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2, 2), (4, 2), (2, 64), (8, 16), (16, 1024), (32, 4), (128, 512), (512, 8), (1024, 2),
                                 (128, 2), (2, 128), (256, 2), (2, 256)])
def test_transform_lengths(W, H):
    i = np.arange(W * H)
    d = ((i * 31 + 7) % 101) - 50.0 + ((i * 13 + 5) % 17) / 17.0
    ref, _ = ffi.poisson(W, H, d, matrix=W * H <= 4096)
    with Placer(P.synthetic(24, 400, 40, 480, 6.0, 0),
                default_params(bins_x=W, bins_y=H, engine=abi.ENGINE_HOST)) as g:
        pot, _ = g.poisson(d)
    assert np.max(np.abs(pot - ref)) <= 1e-6 * np.max(np.abs(ref))


@pytest.mark.parametrize("side,cells,bins_x,bins_y,iterations,stacked", [
    (520, 3000, 512, 512, 2, False), (48, 2000, 64, 32, 4, False), (48, 2000, 16, 8, 4, False),
    (24, 400, 4, 2, 4, False), (96, 9000, 128, 128, 3, False), (140, 18000, 128, 128, 3, False),
    (140, 18000, 128, 64, 3, False), (140, 18000, 256, 64, 3, False), (140, 18000, 64, 256, 3, False),
    (48, 2000, 64, 64, 3, True), (48, 2000, 104, 40, 3, True)])
def test_the_loop_alone_equals_the_loop_in_a_batch(side, cells, bins_x, bins_y, iterations, stacked):
    prob = P.synthetic(side, cells, 60, cells + cells // 5, 6.0, 1)
    if stacked:
        prob.initial_xy[:] = (side // 2, side // 2 + 0.25)
    prm = default_params(best_effort=1, max_iterations=iterations, engine=abi.ENGINE_DEVICE, bins_x=bins_x,
                         bins_y=bins_y)
    t, _, st = Placer(prob, prm).run(allow_nonconverged=True)
    b = Batch(prm)
    assert b.admit(prob, 1)
    got = None
    for _ in range(50):
        b.advance(iterations)
        got = b.retire()
        if got is not None:
            break
    assert got is not None and np.array_equal(got[1], t)
    assert (got[2]["iterations"], got[2]["evaluations"], got[2]["hpwl"]) == (st["iterations"], st["evaluations"], st["hpwl"])


@pytest.mark.parametrize("charge", [1.0, 131071.0, 131072.0, 200000.5])
def test_deposits_that_share_a_bin(charge):
    prob = P.synthetic(48, 700, 40, 840, 6.0, 0)
    prob.member_charge[5::11] = charge
    prm = default_params(target_density=0.9)
    o, g = ffi.Oracle(prob, prm), Placer(prob, prm)
    c, lo, hi = o.initial()
    c = c.reshape(-1, 2)
    at, group = 0, 1
    while at + group < 700:   # groups of 1, 2, ... 32 objects on one point
        c[at:at + group] = (3.25 + group, 40.5 - group)
        at += group
        group = group % 32 + 1
    c = np.clip(c.reshape(-1), lo, hi).astype(np.float32).astype(np.float64)
    phys, fill = g.scatter(c)
    rp, rf, rov, rcnt = o.scatter_fixed(c)
    assert np.array_equal(phys, rp) and np.array_equal(fill, rf)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_coordinates_that_are_not_finite_are_refused(value):
    with Placer(P.synthetic(24, 400, 40, 480, 6.0, 0), default_params()) as g:
        good = np.full(g.n, 11.0)
        before = g.evaluate(good, 4.0)
        for k in (0, g.n // 2, g.n - 1):
            bad = good.copy()
            bad[k] = value
            wag, pot, ev = np.full(2 * g.units, 7.0), np.full(g.num_fields * g.bins, 7.0), abi.Eval()
            code = g.lib.texo_gp_evaluate(g.h, abi.ptr(bad, C.c_double), 4.0, C.byref(ev), abi.ptr(wag, C.c_double), None,
                                          None, abi.ptr(pot, C.c_double))
            assert code == abi.CODE["NONFINITE_UNIT_COORDINATE"]
            assert np.all(wag == 7.0) and np.all(pot == 7.0)
        after = g.evaluate(good, 4.0)
        assert np.array_equal(before["wa_gradient"], after["wa_gradient"])
        assert np.array_equal(before["potential"], after["potential"])


def test_clustering_window_at_the_ends_of_its_intervals():
    count = 40000
    scale = np.sqrt(1e-5 * count) * np.sqrt(2.0)
    reach = 2.5 / np.sqrt(2.0) + 6.0
    ends = np.arange(0, 250) / 32.0
    u = np.concatenate([ends, ends + 1e-9, np.abs(ends - 1e-9), reach + np.array([-1e-3, -1e-9, 0.0, 1e-9, 1e-3, 5.0])])
    n = len(u)
    xy = np.zeros((2 * n, 2))
    xy[0::2] = np.random.default_rng(2).uniform(0, 200, (n, 2))
    xy[1::2] = xy[0::2]
    xy[1::2, 0] += u * scale
    xy[1::2, 1] += u[::-1] * scale * (np.arange(n) % 3 == 0)
    clock_lsr = np.stack([np.repeat(np.arange(n), 2), np.zeros(2 * n, np.int64)], axis=1)
    ce = np.arange(2 * n) % 2
    got, _ = routability.register_clustering_areas(xy, clock_lsr, ce, count)
    code, want = ffi.register_clustering_areas(xy, clock_lsr, ce, count)
    assert code == 0
    assert np.max(np.abs(got - want) / want) <= 1e-12
