"""The work a user has the placement engine do, as timed cases.

Every case goes through the public entry points of texo_gb300 with host
(numpy) arrays, as the C ABI takes them. The netlists are seeded ECP5-like
ones of the benchmark's shape: unit-area cells on a square fabric, fixed IO
evenly spaced on the perimeter, 60 % 2-pin, 30 % 3-5-pin and 10 % 6-32-pin
nets, four of five sinks within a Gaussian radius of the driver's position on
the index grid. The families:

- place      one whole placement call, netlist in, coordinates and targets out
- iterate    a kept handle, restarted and run for some iterations: the device
             engine on a two-kind netlist with macros, timed arcs and fixed
             occupancy on its own tile grid (the reference's default grid),
             or the host engine on a large one-kind netlist, with the FP32 or
             the tensor-core transforms
- evaluate   the objective and its gradients, density and potential at given
             coordinates
- batch      mixed placements resident together until all have converged
- seed       the coarse quadratic seed's linear solve of one axis
- demand     the continuous routing-demand map of the nets' bounding boxes
- clustering the register-clustering areas
- auction    the single-BEL capacity auction of the legalizer
"""
import math

import numpy as np
import torch

from texo_gb300 import abi, legalize, routability
from texo_gb300.placer import Batch, Placer, default_params, place, quadratic_solve, routing_demand
from texo_gb300.problem import Problem


def listed():
    return [
        # the smallest benchmark netlist placed in one call: host model, upload,
        # a hundred short iterations, results; latency counts
        dict(name="place-2k", family="place", cells=2000, side=48, bins=64, density=1.0),
        # the headline size (LFE5U-85), placed in one call
        dict(name="place-42k", family="place", cells=42000, side=210, bins=256, density=0.9),
        # a mapped design with LUT and register kinds, macros, timed arcs and fixed
        # BELs on a tile grid that is no power of two, as a device gives it
        dict(name="iterate-14k-macros", family="iterate", cells=14000, side=104, bins=0, density=1.0, kinds=2,
             engine="device", transform="fp32", iterations=15),
        # the largest benchmark netlist, host engine, FP32 transforms
        dict(name="iterate-1m", family="iterate", cells=1000000, side=1024, bins=1024, density=0.9, kinds=1,
             engine="host", transform="fp32", iterations=3),
        # a quarter of it with the tensor-core transforms
        dict(name="iterate-250k-tensor", family="iterate", cells=250000, side=512, bins=512, density=0.9, kinds=1,
             engine="host", transform="tensor", iterations=4),
        # objective and gradients of a small netlist on its tile grid (a checker's
        # or an outer loop's call): launches and copies count
        dict(name="evaluate-2k", family="evaluate", cells=2000, side=48, bins=0, density=1.0, transform="fp32"),
        # the same at the headline size
        dict(name="evaluate-42k", family="evaluate", cells=42000, side=210, bins=256, density=0.9, transform="fp32"),
        # ECO variants and partitions of many sizes placed together
        dict(name="batch-16", family="batch", jobs=16, smallest=1000, largest=40000),
        # the quadratic seed of the headline netlist, one axis from the centre
        dict(name="seed-42k", family="seed", cells=42000, side=210),
        # the routing-demand map of its nets at spread positions
        dict(name="demand-50k", family="demand", cells=42000, side=210),
        # one register per site of it, 8 control sets, 16 clock enables
        dict(name="clustering-42k", family="clustering", registers=42000, side=210, sets=8, enables=16),
        # its units legalized onto sites
        dict(name="auction-42k", family="auction", cells=42000, side=210, spread=0.4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(n):
    return 1 << (n - 1).bit_length()


def draw(rng):
    family = rng.choice(["place", "iterate", "iterate", "evaluate", "evaluate", "batch", "seed", "demand",
                         "clustering", "auction"])
    if family == "place":
        cells = _log(rng, 1000, 42000)
        side = math.ceil(math.sqrt(cells / rng.uniform(0.8, 0.93)))
        return dict(family=family, cells=cells, side=side, bins=min(256, max(64, _pow2(side))),
                    density=rng.choice([0.95, 1.0]))
    if family == "iterate" and rng.random() < 0.5:
        cells = _log(rng, 2000, 20000)
        return dict(family=family, cells=cells, side=math.ceil(math.sqrt(cells * rng.uniform(0.75, 1.1))), bins=0,
                    density=1.0, kinds=2, engine="device", transform="fp32", iterations=rng.randint(5, 20))
    if family == "iterate":
        bins = rng.choice([256, 512, 1024])
        side = rng.randint(bins * 5 // 8, bins)
        return dict(family=family, cells=int(side * side * rng.uniform(0.7, 0.88)), side=side, bins=bins, density=0.9,
                    kinds=1, engine="host", transform=rng.choice(["fp32", "tensor"]), iterations=rng.randint(2, 3))
    if family == "evaluate":
        cells = _log(rng, 500, 100000)
        side = math.ceil(math.sqrt(cells / rng.uniform(0.75, 0.88)))
        tile = rng.random() < 0.4
        return dict(family=family, cells=cells, side=side, bins=0 if tile else max(64, _pow2(side)), density=0.9,
                    transform="fp32" if tile else rng.choice(["fp32", "tensor"]))
    if family == "batch":
        return dict(family=family, jobs=rng.randint(4, 16), smallest=1000, largest=_log(rng, 4000, 30000))
    if family == "clustering":
        n = _log(rng, 1000, 42000)
        return dict(family=family, registers=n, side=math.ceil(math.sqrt(n / 0.9)), sets=rng.randint(6, 24),
                    enables=rng.randint(1, 32))
    cells = _log(rng, 1000, 100000)
    c = dict(family=family, cells=cells, side=math.ceil(math.sqrt(cells / rng.uniform(0.8, 0.95))))
    if family == "auction":
        c["spread"] = rng.uniform(0.3, 0.5)
    return c


# ---- netlists ---------------------------------------------------------------

def _perimeter(side, count):
    """`count` points evenly spaced along the fabric's perimeter."""
    t = np.arange(count, dtype=np.int64) * (4 * (side - 1)) // count
    leg, at = t // (side - 1), t % (side - 1)
    x = np.choose(leg, [at, np.full_like(at, side - 1), side - 1 - at, np.zeros_like(at)])
    y = np.choose(leg, [np.zeros_like(at), at, np.full_like(at, side - 1), side - 1 - at])
    return np.stack([x, y], axis=1).astype(np.float64)


def _nets(rng, side, cells, io, sigma):
    """(net_ptr, pin_cell): 1.2 nets a cell, driver first, no cell twice in a net."""
    total, count = cells + io, int(1.2 * cells)
    band = rng.random(count)
    degree = np.where(band < 0.6, 2, np.where(band < 0.9, rng.integers(3, 6, count), rng.integers(6, 33, count)))
    net = np.repeat(np.arange(count, dtype=np.int64), degree)
    first = np.cumsum(degree) - degree
    driver = rng.integers(0, total, count)
    at = driver[net]
    x = at % side + np.rint(sigma * rng.standard_normal(net.size)).astype(np.int64)
    y = at // side + np.rint(sigma * rng.standard_normal(net.size)).astype(np.int64)
    near = y * side + x
    local = (rng.random(net.size) < 0.8) & (x >= 0) & (y >= 0) & (x < side) & (y < side) & (near < total)
    pin = np.where(local, near, rng.integers(0, total, net.size))
    pin[first] = driver
    # drop a cell's later pins on the same net, then nets left with one pin
    order = np.argsort(net * total + pin, kind="stable")
    key = (net * total + pin)[order]
    keep = np.ones(net.size, bool)
    keep[order[1:][key[1:] == key[:-1]]] = False
    left = np.bincount(net[keep], minlength=count)
    keep &= left[net] > 1
    left = left[left > 1]
    return np.concatenate([[0], np.cumsum(left)]), pin[keep]


def _netlist(rng, side, cells, start):
    """The arrays of a one-kind netlist; `start`: "centre" (the benchmark's
    jitter around the fabric centre) or "seeded" (spread as a quadratic seed
    leaves the cells)."""
    io = min(4 * (side - 1), max(16, int(1.75 * side)))
    net_ptr, pin_cell = _nets(rng, side, cells, io, 6.0 if side < 128 else 12.0 if side < 384 else 24.0)
    pads = _perimeter(side, io)
    centre, top = 0.5 * (side - 1), float(side - 1)
    spread = 1.0 if start == "centre" else side / 6.0
    xy = np.clip(centre + spread * rng.standard_normal((cells, 2)), 0.0, top)
    return dict(net_ptr=net_ptr, pin_cell=pin_cell, pads=pads, xy=xy, io=io)


def _problem(rng, side, cells, start):
    n = _netlist(rng, side, cells, start)
    io, pads = n["io"], n["pads"]
    total = cells + io
    lower, upper = np.zeros((total, 2)), np.full((total, 2), float(side - 1))
    lower[cells:] = upper[cells:] = pads
    fixed = np.zeros(total, np.uint8)
    fixed[cells:] = 1
    cell_xy = np.zeros((total, 2))
    cell_xy[cells:] = pads
    return Problem(side, side, [(abi.KIND_LUT, 4)], np.ones(side * side, np.uint32), np.concatenate([n["xy"], pads]),
                   lower, upper, np.minimum(np.arange(total + 1), cells), np.zeros(cells, np.uint32),
                   np.zeros((cells, 2)), np.ones(cells), np.arange(cells), np.arange(total), np.zeros((total, 2)),
                   fixed, cell_xy, n["net_ptr"], n["pin_cell"])


def _macro_problem(rng, side, cells):
    """Two kinds (a third of the cells registers), two of five units a macro of
    two cells (a LUT and its register on one site, or a chain of two sites),
    3 % of the BELs held by fixed units, one net in seven with a timed arc."""
    n = _netlist(rng, side, cells, "seeded")
    io, pads = n["io"], n["pads"]
    total = cells + io
    kind = (rng.random(cells) < 0.35).astype(np.int64)
    pair = rng.choice(cells // 2, int(0.57 * (cells // 2)), replace=False) * 2   # cells 2k, 2k + 1 form a macro
    joined = np.zeros(cells, bool)
    joined[pair + 1] = True                                           # the second cell of a macro
    unit = np.cumsum(~joined) - 1                                     # unit of every movable cell
    units = int(unit[-1]) + 1
    offset = np.zeros((total, 2))
    chain = pair[kind[pair] == kind[pair + 1]]
    offset[chain + 1, 1] = 1.0
    top = np.zeros(units)
    top[unit[chain + 1]] = 1.0
    lead = np.flatnonzero(~joined)
    xy = n["xy"][lead].copy()
    xy[:, 1] = np.minimum(xy[:, 1], side - 1 - top)
    lower, upper = np.zeros((units + io, 2)), np.full((units + io, 2), float(side - 1))
    upper[:units, 1] -= top
    lower[units:] = upper[units:] = pads
    fixed = np.zeros(total, np.uint8)
    fixed[cells:] = 1
    cell_xy = np.zeros((total, 2))
    cell_xy[cells:] = pads
    member_ptr = np.concatenate([[0], np.cumsum(np.bincount(unit, minlength=units)), np.full(io, cells)])
    tiles = side * side
    held = np.concatenate([np.stack([np.full(k.size, f), k % side, k // side], axis=1)
                           for f in (0, 1) for k in [rng.choice(tiles, int(0.03 * tiles), replace=False)]])
    ptr, pin = n["net_ptr"], n["pin_cell"]
    timed = np.flatnonzero(rng.random(ptr.size - 1) < 1 / 7)
    sink = pin[ptr[timed] + 1 + (rng.random(timed.size) * (ptr[timed + 1] - ptr[timed] - 1)).astype(np.int64)]
    return Problem(side, side, [(abi.KIND_LUT, 4), (abi.KIND_REGISTER, 0)], np.ones(2 * tiles, np.uint32),
                   np.concatenate([xy, pads]), lower, upper, member_ptr, kind, offset[:cells], np.ones(cells),
                   np.arange(cells), np.concatenate([unit, units + np.arange(io)]), offset, fixed, cell_xy, ptr, pin,
                   pin[ptr[timed]], sink, rng.integers(1, 4, timed.size), fixed_occupancy=held)


def _params(case, engine):
    form = {"fp32": abi.DCT_FP32, "tensor": abi.DCT_TENSOR}[case.get("transform", "fp32")]
    return default_params(bins_x=case["bins"], bins_y=case["bins"], target_density=case["density"],
                          gamma_base=4.0 if case["bins"] else 8.0, max_iterations=1000, best_effort=1,
                          engine=abi.ENGINE_DEVICE if engine == "device" else abi.ENGINE_HOST, dct_mode=form)


def _spread(rng, side, count):
    """Positions of a nearly converged placement: one cell a site, half a tile off."""
    site = rng.permutation(side * side)[:count]
    xy = np.stack([site % side, site // side], axis=1) + 0.5 * rng.standard_normal((count, 2))
    return np.clip(xy, 0.0, side - 1.0)


def _seed_system(rng, side, cells):
    """The bound-to-bound system of one axis at the first linearisation (every
    movable unit at the centre, so every separation counts as one tile): a
    CSR adjacency, fixed pads folded into diagonal and right-hand side, and
    each component without a pad held by its first unit."""
    io = min(4 * (side - 1), max(16, int(1.75 * side)))
    ptr, pin = _nets(rng, side, cells, io, 6.0 if side < 128 else 12.0)
    pad = np.concatenate([np.zeros(cells), _perimeter(side, io)[:, 0]])
    deg = np.diff(ptr)
    net = np.repeat(np.arange(deg.size), deg)
    weight = (64.0 / (deg - 1))[net]
    low, high = pin[ptr[:-1]][net], pin[ptr[1:] - 1][net]
    index = np.arange(pin.size) - ptr[net]
    a = index > 0                                # every other pin to the lower bound
    b = a & (index < (deg - 1)[net])             # every inner pin to the upper bound
    left = np.concatenate([pin[a], pin[b]])
    right = np.concatenate([low[a], high[b]])
    w = np.concatenate([weight[a], weight[b]])
    fixed = np.arange(cells + io) >= cells
    n = cells
    diag = np.zeros(n)
    rhs = np.zeros(n)
    for here, there in ((left, right), (right, left)):
        move = ~fixed[here]
        np.add.at(diag, here[move], w[move])
        held = move & fixed[there]
        np.add.at(rhs, here[held], w[held] * pad[there[held]])
    both = ~fixed[left] & ~fixed[right]
    anchored = np.zeros(n, bool)
    anchored[left[~fixed[left] & fixed[right]]] = True
    anchored[right[~fixed[right] & fixed[left]]] = True
    rows = np.concatenate([left[both], right[both]])
    cols = np.concatenate([right[both], left[both]])
    ws = np.concatenate([w[both], w[both]])
    label = np.arange(n)                         # components by the least unit each can reach
    while True:
        least = label.copy()
        np.minimum.at(least, rows, label[cols])
        least = least[least]
        if np.array_equal(least, label):
            break
        label = least
    has = np.zeros(n, bool)
    has[label[anchored]] = True
    gauge = (label == np.arange(n)) & ~has
    diag[gauge], rhs[gauge] = 1.0, 0.0
    keep = ~gauge[rows] & ~gauge[cols]
    rows, cols, ws = rows[keep], cols[keep], ws[keep]
    order = np.argsort(rows, kind="stable")
    row_ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    start = np.where(gauge, 0.0, 0.5 * (side - 1))
    return dict(diag=diag, ptr=row_ptr, index=cols[order], weight=ws[order], rhs=rhs, start=start)


def _boxes(rng, side, cells):
    """Bounding boxes of a netlist at spread positions: min x, max x, min y, max y."""
    io = min(4 * (side - 1), max(16, int(1.75 * side)))
    ptr, pin = _nets(rng, side, cells, io, 6.0 if side < 128 else 12.0)
    xy = np.concatenate([np.stack([np.arange(cells) % side, np.arange(cells) // side], axis=1)
                         + rng.standard_normal((cells, 2)), _perimeter(side, io)])
    p = np.clip(xy, 0.0, side - 1.0)[pin]
    lo, hi = np.minimum.reduceat(p, ptr[:-1], axis=0), np.maximum.reduceat(p, ptr[:-1], axis=0)
    return np.ascontiguousarray(np.stack([lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1]], axis=1))


def _registers(rng, case):
    xy = _spread(rng, case["side"], case["registers"])
    n = case["registers"]
    control = np.stack([rng.integers(0, case["sets"], n), np.zeros(n, np.int64)], axis=1).astype(np.uint64)
    return xy, control, rng.integers(0, case["enables"], n).astype(np.uint64)


def _coordinates(rng, side, cells, pads, fillers):
    """An optimizer vector near convergence, in the engine's FP32 precision."""
    xy = np.concatenate([_spread(rng, side, cells), pads, rng.uniform(0.0, side - 1.0, (fillers, 2))])
    return xy.astype(np.float32).astype(np.float64).reshape(-1)


GAMMA = 3.0   # wirelength smoothing of the evaluate cases, in tiles


# ---- what a program has in hand, and one pass --------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([seed, 7])
    family = case["family"]
    s = dict(case=case)
    if family == "place":
        s["problem"] = _problem(rng, case["side"], case["cells"], "centre")
        s["params"] = _params(case, "device")
    elif family == "iterate":
        problem = (_macro_problem(rng, case["side"], case["cells"]) if case["kinds"] == 2 else
                   _problem(rng, case["side"], case["cells"], "seeded"))
        s["handle"] = Placer(problem, _params(case, case["engine"]))
    elif family == "evaluate":
        problem = _problem(rng, case["side"], case["cells"], "seeded")
        s["handle"] = h = Placer(problem, _params(case, "host"))
        s["coordinates"] = _coordinates(rng, case["side"], case["cells"], problem.cell_fixed_xy[case["cells"]:],
                                        h.num_fillers)
    elif family == "batch":
        s["jobs"] = []
        for i in range(case["jobs"]):   # sizes spread evenly over their logarithm
            ratio = case["largest"] / case["smallest"]
            cells = int(round(case["smallest"] * ratio ** ((i + 0.5) / case["jobs"])))
            side = math.ceil(math.sqrt(cells / 0.9))
            bins = min(256, max(64, _pow2(side)))
            s["jobs"].append((_problem(rng, side, cells, "centre"),
                              _params(dict(bins=bins, density=1.0), "device")))
    elif family == "seed":
        s["system"] = _seed_system(rng, case["side"], case["cells"])
    elif family == "demand":
        s["boxes"] = _boxes(rng, case["side"], case["cells"])
    elif family == "clustering":
        s["registers"] = _registers(rng, case)
    else:
        side = case["side"]
        # one unit a site, moved by `spread` tiles of noise: how far targets collide
        site = rng.permutation(side * side)[:case["cells"]]
        xy = np.stack([site % side, site // side], axis=1) + case["spread"] * rng.standard_normal((case["cells"], 2))
        s["targets"] = np.clip(np.rint(xy), 0, side - 1).astype(np.uint32)
        s["grid"] = legalize.site_grid(np.ones((side, side), np.uint32))
    return s


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "place":
        targets, coords, stats = place(state["problem"], state["params"], coordinates=True)
        return dict(targets=targets, coordinates=coords, hpwl=stats["hpwl"], overflow=np.array(stats["overflow"]))
    if family == "iterate":
        h = state["handle"]
        h.reset()
        targets, coords, stats = h.run(case["iterations"], allow_nonconverged=True)
        return dict(targets=targets, coordinates=coords, hpwl=stats["hpwl"], overflow=np.array(stats["overflow"]),
                    energy=np.array(stats["energy"]))
    if family == "evaluate":
        e = state["handle"].evaluate(state["coordinates"], GAMMA)
        return dict(wirelength=e["wirelength"], energy=e["fields"][0].energy,
                    overflow=e["fields"][0].normalized_overflow, wa_gradient=e["wa_gradient"],
                    field_gradient=e["field_gradient"], density=e["density"], potential=e["potential"])
    if family == "batch":
        batch = Batch(hbm_budget=64 << 30, max_slots=len(state["jobs"]) + 1)
        for i, (problem, params) in enumerate(state["jobs"]):
            if not batch.admit(problem, i, params):
                raise RuntimeError("the batch refused a job")
        targets, hpwl = [None] * len(state["jobs"]), np.zeros(len(state["jobs"]))
        left = len(state["jobs"])
        while left:
            batch.advance(20)
            while (done := batch.retire()) is not None:
                targets[done[0]], hpwl[done[0]] = done[1], done[2]["hpwl"]
                left -= 1
        batch.close()
        return dict(targets=targets, hpwl=hpwl)
    if family == "seed":
        y = state["system"]
        return quadratic_solve(y["diag"], y["ptr"], y["index"], y["weight"], y["rhs"], y["start"])[0]
    if family == "demand":
        return routing_demand(case["side"], case["side"], state["boxes"])[:2]
    if family == "clustering":
        xy, control, enable = state["registers"]
        return routability.register_clustering_areas(xy, control, enable, 2 * case["registers"])[0]
    result = legalize.auction_singletons(state["grid"], np.zeros(case["cells"], np.uint32), state["targets"])
    return dict(assignment=result.assignment, prices=result.prices)


# ---- the least a pass moves and computes --------------------------------------

def _placement_work(cells, side, bins, kinds, evaluations, iterations):
    """Bytes and operations of an iteration loop with the given evaluations of
    the whole objective: members and fillers read, grids written and read once,
    pins and nets read, gradients written, and per iteration the optimizer's
    vectors; a transform counts 5 n log2 n operations a grid four times."""
    b = float(bins or side) ** 2
    pins, nets, fillers = 5.3 * cells, 1.2 * cells, float(side) ** 2 * kinds
    objects = cells + fillers
    per_eval = 20 * cells + 16 * fillers + 16 * kinds * b + 12 * pins + 8 * nets + 24 * objects
    per_step = 60 * objects
    flops = 60 * objects + 40 * pins + 4 * 5 * kinds * b * math.log2(max(b, 2))
    return evaluations * per_eval + iterations * per_step, evaluations * flops


def work(case):
    family = case["family"]
    if family == "place":
        moved, flops = _placement_work(case["cells"], case["side"], case["bins"], 1, 185, 80)
    elif family == "iterate":
        k = case["iterations"]
        moved, flops = _placement_work(case["cells"], case["side"], case["bins"], case["kinds"], 2.3 * k + 1, k)
    elif family == "evaluate":
        moved, flops = _placement_work(case["cells"], case["side"], case["bins"], 1, 1, 0)
        moved += 8 * (6 * case["cells"] + 4 * case["side"] ** 2 + 2 * (case["bins"] or case["side"]) ** 2)
    elif family == "batch":
        lo, hi = math.log(case["smallest"]), math.log(case["largest"])
        mean = (case["largest"] - case["smallest"]) / (hi - lo) if hi > lo else case["largest"]
        side = math.ceil(math.sqrt(mean / 0.9))
        moved, flops = _placement_work(mean, side, max(64, _pow2(side)), 1, 185 * case["jobs"], 80 * case["jobs"])
    elif family == "seed":
        entries, n = 12.5 * case["cells"], float(case["cells"])
        moved, flops = 60 * (12 * entries + 100 * n), 60 * (2 * entries + 13 * n)
    elif family == "demand":
        boxes, tiles = 1.2 * case["cells"], float(case["side"]) ** 2
        moved, flops = 32 * boxes + 16 * tiles, 80 * boxes + 4 * tiles
    elif family == "clustering":
        n = float(case["registers"])
        sigma = math.sqrt(1e-5 * 2 * n)
        reach = min(1.0, (2 * 10.9 * sigma / case["side"]) ** 2)
        pairs = n * n / case["sets"] * reach
        moved, flops = 40 * n, 4 * 40 * pairs
    else:
        n, tiles = float(case["cells"]), float(case["side"]) ** 2
        moved, flops = 16 * n + 8 * tiles, 60 * n
    return dict(bytes=moved, flops=flops)


# ---- the same values in 64 bits ------------------------------------------------

def _taps(coordinate, bins):
    """Quadratic B-spline stencil on a clamped axis: bin indices, weights and
    derivative weights [n, 3]."""
    c = np.clip(coordinate, 0.0, bins - 1.0)
    centre = np.minimum(np.floor(c + 0.5), bins - 1.0)
    o = c - centre
    i = centre.astype(np.int64)
    index = np.stack([np.maximum(i - 1, 0), i, np.minimum(i + 1, bins - 1)], axis=1)
    weight = np.stack([0.5 * (0.5 - o) ** 2, 0.75 - o * o, 0.5 * (0.5 + o) ** 2], axis=1)
    return index, weight, np.stack([o - 0.5, -2.0 * o, o + 0.5], axis=1)


def _exact_evaluate(case, seed):
    rng = np.random.default_rng([seed, 7])
    side, cells = case["side"], case["cells"]
    n = _netlist(rng, side, cells, "seeded")
    io, ptr, pin = n["io"], n["net_ptr"], n["pin_cell"]
    bins = case["bins"] or side
    scale = bins / side
    tiles = side * side
    total = case["density"] * tiles - cells
    fillers = tiles if total > 0 else 0
    at = _coordinates(rng, side, cells, n["pads"], fillers).reshape(-1, 2)
    to_bins = (lambda v: v) if bins == side else (lambda v: (v + 0.5) * scale - 0.5)

    def spread(xy, charge):
        ix, wx, _ = _taps(to_bins(xy[:, 0]), bins)
        iy, wy, _ = _taps(to_bins(xy[:, 1]), bins)
        tap = charge[:, None, None] * wy[:, :, None] * wx[:, None, :]
        return np.bincount((iy[:, :, None] * bins + ix[:, None, :]).ravel(), tap.ravel(), bins * bins)

    # density: cells minus the smoothed capacity, then the fillers
    site = np.stack([np.arange(tiles) % side, np.arange(tiles) // side], axis=1).astype(np.float64)
    physical = spread(at[:cells], np.ones(cells)) - spread(site, np.full(tiles, case["density"]))
    charge = np.full(fillers, total / tiles)
    density = physical + (spread(at[cells + io:], charge) if fillers else 0.0)
    # potential: the orthonormal cosine basis and the 5-point Laplacian's eigenvalues
    k = np.arange(bins)
    basis = np.cos(np.pi * k[:, None] * (k[None, :] + 0.5) / bins) * np.sqrt(2.0 / bins)
    basis[0] = math.sqrt(1.0 / bins)
    eigen = 4.0 * np.sin(np.pi * k / (2.0 * bins)) ** 2
    eigen = eigen[:, None] + eigen[None, :]
    eigen[0, 0] = 1.0
    centred = (density - density.mean()).reshape(bins, bins)
    modes = basis @ centred @ basis.T / eigen
    modes[0, 0] = 0.0
    potential = basis.T @ modes @ basis
    # field gradient of every cell and filler
    gradient = np.zeros((cells + io + fillers, 2))
    for lo, hi, q in ((0, cells, np.ones(cells)), (cells + io, cells + io + fillers, charge)):
        ix, wx, dx = _taps(to_bins(at[lo:hi, 0]), bins)
        iy, wy, dy = _taps(to_bins(at[lo:hi, 1]), bins)
        v = potential[iy[:, :, None], ix[:, None, :]]
        step = 1.0 if bins == side else scale
        gradient[lo:hi, 0] = q * step * np.einsum("nrc,nr,nc->n", v, wy, dx)
        gradient[lo:hi, 1] = q * step * np.einsum("nrc,nr,nc->n", v, dy, wx)
    # weighted-average wirelength
    xy = np.concatenate([at[:cells], n["pads"]])[pin]
    net = np.repeat(np.arange(ptr.size - 1), np.diff(ptr))
    wa_gradient = np.zeros((cells + io, 2))
    wirelength = 0.0
    for axis in (0, 1):
        v = xy[:, axis]
        per_pin = np.zeros(v.size)
        for sign in (1.0, -1.0):
            far = np.maximum.reduceat(sign * v, ptr[:-1])
            d = sign * v - far[net]
            w = np.exp(d / GAMMA)
            sum_w = np.add.reduceat(w, ptr[:-1])
            mean = np.add.reduceat(w * d, ptr[:-1]) / sum_w
            wirelength += float(np.sum(far + mean))
            per_pin += sign * w / sum_w[net] * (1.0 + (d - mean[net]) / GAMMA)
        wa_gradient[:, axis] = np.bincount(pin, per_pin, cells + io)
    wa_gradient[cells:] = 0.0
    return dict(wirelength=wirelength, energy=0.5 * float(np.sum(centred * potential)),
                overflow=float(np.sum(np.maximum(physical, 0.0))) / cells, wa_gradient=wa_gradient.reshape(-1),
                field_gradient=gradient.reshape(1, -1), density=density.reshape(1, -1),
                potential=potential.reshape(1, -1))


def _exact_seed(y):
    """The system solved to rounding: conjugate gradients on D^-1/2 (D - W) D^-1/2."""
    n = y["diag"].size
    row = np.repeat(np.arange(n), np.diff(y["ptr"]))

    def times(v):
        return y["diag"] * v - np.bincount(row, y["weight"] * v[y["index"]], n)

    x = y["start"].copy()
    r = y["rhs"] - times(x)
    z = r / y["diag"]
    p, rz, stop = z.copy(), float(r @ z), 1e-26 * max(float(r @ z), 1e-300)
    for _ in range(2000):
        if rz <= stop:
            break
        q = times(p)
        alpha = rz / float(p @ q)
        x += alpha * p
        r -= alpha * q
        z = r / y["diag"]
        rz, old = float(r @ z), rz
        p = z + rz / old * p
    return x


def _exact_demand(case, boxes):
    """Every box spread over the tiles it overlaps after half a tile of margin."""
    side = case["side"]
    x0, x1, y0, y1 = boxes.T
    area = (x1 - x0 + 1.0) * (y1 - y0 + 1.0)
    tile = torch.arange(side, dtype=torch.float64)
    out = [torch.zeros(side, side, dtype=torch.float64) for _ in range(2)]
    for at in range(0, boxes.shape[0], 8192):
        part = slice(at, at + 8192)

        def cover(lo, hi):
            a, b = torch.from_numpy(lo[part].copy())[:, None], torch.from_numpy(hi[part].copy())[:, None]
            return (torch.minimum(tile + 0.5, b + 0.5) - torch.maximum(tile - 0.5, a - 0.5)).clamp(min=0.0)

        cx, cy = cover(x0, x1), cover(y0, y1)
        for k, span in enumerate((x1 - x0, y1 - y0)):
            out[k] += (cy * torch.from_numpy((span / area)[part].copy())[:, None]).T @ cx
    return tuple(v.numpy() for v in out)


def _exact_clustering(case, registers):
    xy, control, enable = registers
    sigma = math.sqrt(1e-5 * 2 * case["registers"])
    half, scale = 2.5 * sigma, sigma * math.sqrt(2.0)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    areas = np.zeros(case["registers"])

    def ceiling(v, d):
        q = v / d
        f = torch.floor(q)
        return torch.where(q - f < 1.0 / d, v + (1.0 - d) * f, torch.ceil(q))

    for group in np.unique(control[:, 0]):
        who = np.flatnonzero(control[:, 0] == group)
        pos = torch.from_numpy(xy[who]).to(device)
        ce = torch.from_numpy(enable[who].astype(np.int64)).to(device)
        names, ce = torch.unique(ce, return_inverse=True)
        member = torch.nn.functional.one_hot(ce, names.numel()).double()
        for at in range(0, who.size, 2048):
            rows = slice(at, at + 2048)
            p = 1.0
            for axis in (0, 1):
                d = pos[rows, axis][:, None] - pos[None, :, axis]
                p = p * (0.5 * (torch.erf((d + half) / scale) - torch.erf((d - half) / scale))).clamp(0.0, 1.0)
            expected = p @ member
            focal = expected.gather(1, ce[rows][:, None])[:, 0]
            total = ceiling(expected, 2.0).sum(dim=1)
            areas[who[rows]] = (8.0 / focal * ceiling(focal, 2.0) / total * ceiling(total, 4.0)).cpu().numpy()
    return areas


def exact(case, seed):
    family = case["family"]
    if family == "evaluate":
        return _exact_evaluate(case, seed)
    rng = np.random.default_rng([seed, 7])
    if family == "seed":
        return _exact_seed(_seed_system(rng, case["side"], case["cells"]))
    if family == "demand":
        return _exact_demand(case, _boxes(rng, case["side"], case["cells"]))
    if family == "clustering":
        return _exact_clustering(case, _registers(rng, case))
    # placements follow a line search from iteration to iteration: no closed value
    return None
