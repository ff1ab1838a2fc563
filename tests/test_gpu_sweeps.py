"""The wavefront sweeps of the plain form at the edges of their tiles: IC(0) and the
multigrid cycle, bit for bit the oracle's natural-order loops (8x8 tiles of x-pencils:
remainders in y and z, pencils shorter than the tile's skew and longer than the ring of
received values, per-face weights, right-hand sides outside the range of the division from
precomputed reciprocals)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float64).view(np.uint64)


@pytest.mark.parametrize("scale", [1.0, 1e-290])
@pytest.mark.parametrize("faces", ["uniform", "perturbed"])
@pytest.mark.parametrize("cells", [(2, 9, 7), (3, 8, 8), (17, 17, 9), (300, 5, 3), (21, 24, 16)])
def test_sweeps_bitwise_at_tile_edges(pkg, O, cells, faces, scale):
    boxes = [((3.0, 3.0, 0.0), (7.5, 7.5, 4.5))] if min(cells) > 8 else []
    case = pkg.synth.case(cells, 1.5, inflow=5.0, boxes=boxes)
    g = pkg.grid.Grid.build(case)
    og = O.Grid(case)
    dg = pkg.pressure.DeviceGrid(g, preconditioner="ic0")
    if faces == "perturbed":
        area = g.face_area * (1.0 + (np.arange(g.n_faces) % 7) * 0.025)
        og.set_faces(area=area)
        dg.update_faces(area=area)
    rng = np.random.default_rng(sum(cells))
    r = np.where(g.fluid == 1, rng.uniform(-1.0, 1.0, g.count), 0.0)
    r[rng.integers(0, g.count, g.count // 8)] = 0.0
    r *= scale
    for _ in range(2):  # a second sweep over the same hand-off entries
        assert np.array_equal(bits(dg.precondition(r)), bits(og.ic0_apply(r)))
    dg.configure("multigrid")
    og.set_preconditioner("multigrid")
    oz, _ = og.mg_apply(r)
    for _ in range(2):
        assert np.array_equal(bits(dg.precondition(r)), bits(oz))
    dg.close()


@pytest.mark.parametrize("cells, boxes", [((100, 92, 50), 6), ((60, 44, 24), 0), ((75, 61, 37), 4), ((34, 30, 18), 2)])
def test_coarse_cluster_cycle_bitwise(pkg, O, cells, boxes):
    """The plain cycle's coarse levels on one thread-block cluster: a first coarse level whose
    transfers are grid-wide, the 27-point levels of a grid without solid cells, levels split
    over the blocks and levels of one block, each cycle the oracle's bits."""
    rng = np.random.default_rng(cells[0])
    case = pkg.synth.case(cells, 2.0, inflow=5.0, preconditioner="multigrid",
                          boxes=pkg.synth.random_boxes(rng, boxes, [2.0 * v for v in cells], side=(8.0, 24.0), dx=2.0))
    g = pkg.grid.Grid.build(case)
    og = O.Grid(case)
    dg = pkg.pressure.DeviceGrid(g, preconditioner="multigrid")
    for seed in range(2):
        r = np.where(g.fluid == 1, np.random.default_rng(seed).uniform(-1.0, 1.0, g.count), 0.0)
        oz, _ = og.mg_apply(r)
        assert np.array_equal(bits(dg.precondition(r)), bits(oz))
    dg.close()


def test_cycle_within_small_budgets(pkg, O):
    """A context too small for the coarse levels' plan as well still takes the grid, with the
    same bits: budgets from ample down to the smallest that admits it."""
    case = pkg.synth.case((60, 44, 24), 2.0, inflow=5.0, preconditioner="multigrid",
                          boxes=[((20.0, 20.0, 0.0), (42.0, 44.0, 18.0)), ((70.0, 50.0, 0.0), (84.0, 70.0, 30.0))])
    g = pkg.grid.Grid.build(case)
    r = np.where(g.fluid == 1, np.random.default_rng(3).uniform(-1.0, 1.0, g.count), 0.0)
    oz, _ = O.Grid(case).mg_apply(r)
    lo, hi, held = 0, 1 << 28, set()
    while hi - lo > 1 << 10:
        mid = (lo + hi) // 2
        ctx = pkg.pressure.Context(0, hbm_budget_bytes=mid)
        try:
            dg = pkg.pressure.DeviceGrid(g, ctx=ctx, preconditioner="multigrid")
            try:
                assert np.array_equal(bits(dg.precondition(r)), bits(oz))
                held.add(dg.multigrid_stats()["allocated_bytes"])
                hi = mid
            finally:
                dg.close()
        except pkg.pressure.PressureError as e:
            assert "budget" in str(e)
            lo = mid
        ctx.close()
    assert len(held) == 2, held  # with the plan and without


@pytest.mark.parametrize("cells, size", [
    ((9, 7, 100), (9.0, 7.0, 2.0)),      # more rows per line than two per lane
    ((70, 72, 5), (70.0, 72.0, 0.5)),    # more lines per dependency level than warps
    ((5, 5, 400), (5.0, 5.0, 8.0)),      # records too long to copy ahead
    ((24, 4, 4), (240.0, 4.0, 4.0)),     # blocks of a whole plane
    ((470, 460, 2), (470.0, 460.0, 0.2)),  # iterate beyond the cluster's shared memory
])
@pytest.mark.parametrize("boundaries", [("open", "wall", "wall"), ("open", "periodic", "wall")])
def test_line_sweeps_bitwise(pkg, O, cells, size, boundaries):
    """Block Gauss-Seidel sweeps of anisotropic grids on a cluster, each cycle the oracle's bits."""
    if boundaries[1] == "periodic" and cells[0] > 100:
        pytest.skip("the large grid once")
    case = pkg.synth.case(cells, 1.0, boundaries=boundaries, inflow=1.0, preconditioner="multigrid")
    case["domain"]["size_m"] = list(size)
    g = pkg.grid.Grid.build(case)
    og = O.Grid(case)
    dg = pkg.pressure.DeviceGrid(g, preconditioner="multigrid")
    for seed in range(2):
        r = np.random.default_rng(seed).uniform(-1.0, 1.0, g.count)
        oz, _ = og.mg_apply(r)
        assert np.array_equal(bits(dg.precondition(r)), bits(oz))
    assert dg.multigrid_stats()["block_smoothers"]
    dg.close()


def center_of(x):
    """x less its mean in the engine's order: 256 strided sums, trees over 32 lanes and 8 warps."""
    acc = np.zeros(256)
    for k in range(0, x.size, 256):
        acc[:x[k:k + 256].size] += x[k:k + 256]
    w = acc.reshape(8, 32)
    while w.shape[1] > 1:
        w = w[:, :w.shape[1] // 2] + w[:, w.shape[1] // 2:]
    w = w[:, 0]
    while w.size > 1:
        w = w[:w.size // 2] + w[w.size // 2:]
    return x - w[0] / x.size


@pytest.mark.parametrize("cells", [(89, 23, 1), (32, 8, 8), (683, 3, 1), (64, 64, 2), (67, 43, 29)])
def test_center_bitwise(pkg, cells):
    """The gauge of a closed grid in one launch and in two (2,048 members and more), with
    members that fill the last stretch of loads and that do not."""
    g = pkg.grid.Grid.build(pkg.synth.case(cells, 1.0, boundaries=("wall", "wall", "wall"), inflow=0.0))
    dg = pkg.pressure.DeviceGrid(g, preconditioner="ic0")
    x = np.random.default_rng(cells[0]).uniform(-1.0, 1.0, g.count) + 0.5
    want = center_of(x)
    dg.center_nullspaces(x)
    assert np.array_equal(bits(x), bits(want))
    dg.close()


@pytest.mark.parametrize("muscl", [False, True])
@pytest.mark.parametrize("cells, dx", [((31, 8, 5), 2.0), ((33, 9, 4), 1.5), ((64, 7, 3), 1.9), ((95, 17, 2), 2.3),
                                       ((2, 40, 37), 0.3), ((160, 130, 23), 1.3)])
def test_scalar_pass_bitwise_at_tile_edges(pkg, O, cells, dx, muscl):
    """The scalar passes at the edges of their 32 x 8 tiles, shares of a column's slices and
    end faces of less than four slices, with spacings whose quotients go through the exponent
    field, a reciprocal and a reciprocal with the extra correction: the oracle's bits."""
    torch = pytest.importorskip("torch")
    case = pkg.synth.case(cells, dx, inflow=2.0, preconditioner="multigrid",
                          boxes=[] if min(cells) < 5 else [((4 * dx, 2 * dx, 0.0), (9 * dx, 5 * dx, 3 * dx))])
    g = pkg.grid.Grid.build(case)
    og = O.Grid(case)
    rng = np.random.default_rng(sum(cells))
    open_ = np.isin(g.face_kind, (pkg.grid.INTERIOR, pkg.grid.INLET, pkg.grid.OUTLET))
    u = np.where(open_, rng.uniform(-2.0, 2.0, g.n_faces), 0.0)
    fluid = g.fluid.astype(bool)
    c = np.where(fluid & (rng.uniform(size=g.count) < 0.7), rng.uniform(0.0, 1e-3, g.count), 0.0)
    d = np.where(fluid, rng.uniform(0.01, 0.5, g.count), 0.0)
    source = np.where(rng.uniform(size=g.count) < 0.01, 1e-3, 0.0)
    dg = pkg.pressure.DeviceGrid(g, preconditioner="multigrid")
    dg.set_advection("muscl" if muscl else "linear_upwind")
    d_u, d_c, d_d, d_s = (torch.from_numpy(v.copy()).cuda() for v in (u, c, d, source))
    ref = c
    for _ in range(2):
        ref = og.scalar_step(ref, u, d, source, 0.01, muscl=muscl)
        dg.scalar_step_device(d_u.data_ptr(), d_c.data_ptr(), d_d.data_ptr(), d_s.data_ptr(), 0.01)
        torch.cuda.synchronize()
        assert np.array_equal(bits(d_c.cpu().numpy()), bits(ref))
    dg.close()
