"""Device memory of a grid: contexts with just the bytes that a grid once needed still take it,
with the bits of an ample context. What makes the kernels fast but can be left out (plans of the
coarse levels, records of the block smoothers) must never be what a grid is refused for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALLS = ("wall", "wall", "wall")


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.uint64)


def iso(pkg, n, dx=2.0, nb=0, boundaries=("open", "slip", "slip"), inflow=5.0, boxes=()):
    boxes = boxes or pkg.synth.random_boxes(np.random.default_rng(1), nb, [dx * v for v in n], side=(3 * dx, 8 * dx), dx=dx)
    return pkg.synth.case(n, dx, boundaries=boundaries, inflow=inflow, preconditioner="multigrid", boxes=boxes)


PLAIN = {  # case, preconditioner, bytes
    "ic0 periodic": (dict(n=(20, 12, 12), boundaries=("open", "periodic", "wall")), "ic0", 863108),
    "one level": (dict(n=(4, 4, 2)), "multigrid", 28852),
    "one layer": (dict(n=(64, 48, 1)), "multigrid", 1696768),
    "one tile, long pencils": (dict(n=(400, 2, 2)), "multigrid", 916396),
    "two tiles, long pencils": (dict(n=(1000, 9, 2)), "multigrid", 9276834),
    "small": (dict(n=(12, 10, 8)), "multigrid", 463372),
    "open": (dict(n=(60, 44, 24)), "multigrid", 35671860),
    "closed": (dict(n=(64, 48, 32), boundaries=WALLS, inflow=0.0), "multigrid", 56836344),
    "closed, buildings": (dict(n=(64, 48, 32), boundaries=WALLS, inflow=0.0, nb=3), "multigrid", 28841396),
    "periodic": (dict(n=(48, 40, 24), boundaries=("open", "periodic", "wall")), "multigrid", 30163932),
    "periodic, buildings": (dict(n=(48, 40, 24), boundaries=("open", "periodic", "wall"), nb=3), "multigrid", 16715900),
}


@pytest.mark.parametrize("name", list(PLAIN))
def test_plain_form_within_the_bytes(pkg, name):
    kw, pre, held = PLAIN[name]
    g = pkg.grid.Grid.build(iso(pkg, **kw))
    r = np.where(np.asarray(g.fluid) == 1, np.random.default_rng(3).uniform(-1.0, 1.0, g.count), 0.0)
    out = []
    for budget in (1 << 36, held):
        ctx = pkg.pressure.Context(0, hbm_budget_bytes=budget)
        dg = pkg.pressure.DeviceGrid(g, ctx=ctx, preconditioner=pre)
        out.append([dg.precondition(r) for _ in range(2)])
        dg.close()
        ctx.close()
    assert np.array_equal(bits(out[0]), bits(out[1]))


THIN = {  # cells, size, boundaries, bytes
    "lines": ((48, 48, 48), (1.0, 1.0, 0.1), ("open", "wall", "wall"), 105091160),
    "folded lines, closed": ((48, 48, 48), (1.0, 1.0, 0.1), ("wall", "periodic", "wall"), 106928508),
    "long lines": ((9, 7, 100), (9.0, 7.0, 2.0), ("open", "wall", "wall"), 5974167),
    "many lines": ((70, 72, 5), (70.0, 72.0, 0.5), ("open", "wall", "wall"), 24348898),
    "records not copied ahead": ((5, 5, 400), (5.0, 5.0, 8.0), ("open", "wall", "wall"), 9323877),
    "planes": ((24, 4, 4), (240.0, 4.0, 4.0), ("open", "wall", "wall"), 259812),
    "single rows": ((40, 30, 1), (40.0, 30.0, 0.05), ("open", "wall", "wall"), 850766),
    "lines beyond the shared memory": ((3, 3, 7000), (3.0, 3.0, 35.0), ("open", "wall", "wall"), 55920741),
}


@pytest.mark.parametrize("name", list(THIN))
def test_anisotropic_grids_within_the_bytes(pkg, name):
    cells, size, boundaries, held = THIN[name]
    case = pkg.synth.case(cells, 1.0, boundaries=boundaries, inflow=1.0 if boundaries[0] == "open" else 0.0,
                          preconditioner="multigrid")
    case["domain"]["size_m"] = list(size)
    g = pkg.grid.Grid.build(case)
    r = np.random.default_rng(3).uniform(-1.0, 1.0, g.count)
    out = []
    for budget in (1 << 36, held):
        ctx = pkg.pressure.Context(0, hbm_budget_bytes=budget)
        dg = pkg.pressure.DeviceGrid(g, ctx=ctx, preconditioner="multigrid")
        out.append([dg.precondition(r) for _ in range(2)])
        dg.close()
        ctx.close()
    assert np.array_equal(bits(out[0]), bits(out[1]))


def test_more_dependency_levels_than_shared_memory_holds(pkg, O):
    """A duct of 60,000 cells: more dependency levels of its lines than a record sweep keeps starts of."""
    case = pkg.synth.case((60000, 2, 2), 1.0, boundaries=("open", "wall", "wall"), inflow=1.0, preconditioner="multigrid")
    case["domain"]["size_m"] = [60000.0, 2.0, 0.2]
    g = pkg.grid.Grid.build(case)
    r = np.random.default_rng(3).uniform(-1.0, 1.0, g.count)
    oz, _ = O.Grid(case).mg_apply(r)
    dg = pkg.pressure.DeviceGrid(g, preconditioner="multigrid")
    assert np.array_equal(bits(dg.precondition(r)), bits(oz))
    dg.close()


MIXED = {  # cases of a batch, bytes
    "smallest": ([dict(n=(4, 4, 4))], 45100),
    "small": ([dict(n=(8, 8, 8))], 284888),
    "odd rows": ([dict(n=(9, 7, 8))], 299703),
    "no solid cell": ([dict(n=(60, 44, 24))], 40386560),
    "mostly solid": ([dict(n=(45, 39, 21), boxes=[((8.0, 0.0, 0.0), (90.0, 70.0, 42.0))])], 11026432),
    "buildings": ([dict(n=(37, 29, 33), dx=1.5, nb=3)], 12873728),
    "closed": ([dict(n=(64, 48, 32), boundaries=WALLS, inflow=0.0, nb=3)], 37371904),
    "five smallest": ([dict(n=(4, 4, 4))] * 5, 223148),
    "two without solid cells": ([dict(n=(40, 44, 24)), dict(n=(33, 30, 17))], 37535744),
}


def mixed(pkg, grids, budget):
    """Projections of the grids alone, or of several in a batch; also what ran the coarse levels."""
    us = [pkg.synth.random_velocity(g, 70 + i) for i, g in enumerate(grids)]
    ps = [np.zeros(g.count) for g in grids]
    ctx = pkg.pressure.Context(0, hbm_budget_bytes=budget)
    dgs, batch = [], None
    try:
        for g in grids:
            dgs.append(pkg.pressure.DeviceGrid(g, ctx=ctx, preconditioner="multigrid", precision="mixed"))
        batch = pkg.pressure.Batch(dgs, ctx=ctx)
        kernel = batch.stats()["coarse_kernel"]
        if len(dgs) > 1:
            assert all(code == 0 for code, _ in batch.project(us, ps, [0.1] * len(grids), 1e-8, 10000))
        else:
            batch.close()
            batch = None
            dgs[0].project(us[0], ps[0], 0.1, 1e-8, 10000)
    finally:
        if batch:
            batch.close()
        for d in dgs:
            d.close()
        ctx.close()
    return [bits(a) for a in us + ps], kernel


@pytest.mark.parametrize("name", list(MIXED))
def test_mixed_form_within_the_bytes(pkg, name):
    cases, held = MIXED[name]
    grids = [pkg.grid.Grid.build(iso(pkg, **kw)) for kw in cases]
    ample, _ = mixed(pkg, grids, 1 << 36)
    least, _ = mixed(pkg, grids, held)
    assert all(np.array_equal(a, b) for a, b in zip(ample, least))


def test_mixed_form_without_its_plans(pkg):
    """Budgets from ample down to the least that admits the grid: some without room for the cluster's plan."""
    grids = [pkg.grid.Grid.build(iso(pkg, n=(37, 29, 33), dx=1.5, nb=3))]
    ample, kernel = mixed(pkg, grids, 1 << 36)
    lo, hi, seen = 0, 1 << 24, {kernel}
    while hi - lo > 1 << 8:
        mid = (lo + hi) // 2
        try:
            out, kernel = mixed(pkg, grids, mid)
        except pkg.pressure.PressureError as e:
            assert "budget" in str(e)
            lo = mid
            continue
        assert all(np.array_equal(a, b) for a, b in zip(ample, out))
        seen.add(kernel)
        hi = mid
    assert seen == {"cluster", "cooperative"}


@pytest.mark.parametrize("form", ["plain", "lines", "mixed beside plain"])
def test_several_grids_within_the_bytes(pkg, form):
    """Three grids in a context of three times the bytes of one: what an earlier grid holds beyond them
    gives way to a later one, whichever is used, and in turns."""
    if form == "lines":
        cells, size, boundaries, held = THIN["long lines"]
        case = pkg.synth.case(cells, 1.0, boundaries=boundaries, inflow=1.0, preconditioner="multigrid")
        case["domain"]["size_m"] = list(size)
        total = 3 * held
    else:
        case = iso(pkg, n=(60, 44, 24))
        total = 3 * PLAIN["open"][2]
    if form == "mixed beside plain":
        total = 2 * PLAIN["open"][2] + MIXED["no solid cell"][1]
    g = pkg.grid.Grid.build(case)
    rs = [np.random.default_rng(s).uniform(-1.0, 1.0, g.count) for s in range(3)]
    u = pkg.synth.random_velocity(g, 70)
    out = []
    for budget in (1 << 36, total):
        ctx = pkg.pressure.Context(0, hbm_budget_bytes=budget)
        dgs, got = [], []
        for i in range(3):
            mixed_one = form == "mixed beside plain" and i == 2
            dgs.append(pkg.pressure.DeviceGrid(g, ctx=ctx, preconditioner="multigrid",
                                               precision="mixed" if mixed_one else "plain"))
            if mixed_one:
                uu, pp = u.copy(), np.zeros(g.count)
                dgs[i].project(uu, pp, 0.1, 1e-8, 1000)
                got += [uu, pp]
            else:
                got.append(dgs[i].precondition(rs[i]))
        for _ in range(2):
            got += [d.precondition(r) for d, r in list(zip(dgs, rs))[:2]]
        for d in dgs:
            d.close()
        ctx.close()
        out.append([bits(a) for a in got])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
