"""Device memory of a grid: contexts with just the bytes that a grid once needed still take it,
with the bits of an ample context. What makes the kernels fast but can be left out (plans of the
coarse levels, records of the block smoothers) must never be what a grid is refused for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WALLS = ("wall", "wall", "wall")


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.uint64)


def iso(pkg, n, dx=2.0, nb=0, boundaries=("open", "slip", "slip"), inflow=5.0):
    boxes = pkg.synth.random_boxes(np.random.default_rng(1), nb, [dx * v for v in n], side=(3 * dx, 8 * dx), dx=dx)
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
