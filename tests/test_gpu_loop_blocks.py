"""The on-chip loop with other block counts: off, a few blocks, and more blocks than
the device holds at once, which the runtime refuses before the launch starts; such a
run, its snapshots and a batch go through the step kernels. All the same bits."""
import numpy as np
import pytest

import test_gpu_loop2d as loop2d

pytestmark = pytest.mark.gpu


def _plan(pkg, ctx, grid, precision):
    s = loop2d._setup(pkg, grid, precision, seed=grid[0])
    return s, ctx.plan(s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"])


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_fewer_blocks(pkg, precision):
    ctx = pkg.Context(0)
    _, plan = _plan(pkg, ctx, (409, 333, 20, False), precision)
    ctx.set_loop_blocks(0)
    assert plan.route() == 0 and plan.launch_count() == loop2d.NT
    plan.run()
    traces, field = plan.traces(), plan.field()
    for blocks in (-1, 37, 24, -1):
        ctx.set_loop_blocks(blocks)
        plan.reset()
        assert plan.route() == pkg._lib.ROUTE_LOOP
        plan.run(23)
        plan.run()
        np.testing.assert_array_equal(plan.traces(), traces)
        np.testing.assert_array_equal(plan.field(), field)
    ctx.set_loop_blocks(1)  # too large for one block
    plan.reset()
    assert plan.route() == 0
    plan.close()
    ctx.close()


def test_refused_launch_goes_step_by_step(pkg):
    ctx = pkg.Context(0)
    s, plan = _plan(pkg, ctx, (2083, 1019, 20, True), "f64")  # full blocks at 296 tiles
    assert plan.route() == pkg._lib.ROUTE_STRIPS
    plan.run()
    traces, field = plan.traces(), plan.field()
    plan.reset()
    shots = plan.run_snapshots(24, 12)
    plan.close()
    ctx.set_loop_blocks(296)
    _, plan = _plan(pkg, ctx, (2083, 1019, 20, True), "f64")
    assert plan.route() == pkg._lib.ROUTE_LOOP
    plan.run()
    np.testing.assert_array_equal(plan.traces(), traces)
    np.testing.assert_array_equal(plan.field(), field)
    plan.reset()
    assert plan.route() == pkg._lib.ROUTE_STRIPS  # refused, and remembered
    plan.close()
    _, plan = _plan(pkg, ctx, (2083, 1019, 20, True), "f64")
    for a, b in zip(plan.run_snapshots(24, 12), shots):
        np.testing.assert_array_equal(a, b)
    plan.close()
    p = s["problem"]
    model = pkg.Problem(ndim=2, precision=p.precision, nx=p.nx, ny=p.ny, nz=1, halo=p.halo,
                        freetop=p.freetop, dx=p.dx, dy=p.dy, dz=1.0, dt=p.dt, nt=p.nt, nsrc=0,
                        nrec=0)
    batch = pkg.Batch(ctx, [model], [s["vel"]], [s], [0])
    assert batch.launch_count() == 1
    batch.run()
    np.testing.assert_array_equal(batch.traces(0), traces)
    batch.reset()
    assert batch.launch_count() == loop2d.NT
    batch.autotune(4)
    batch.run()
    np.testing.assert_array_equal(batch.traces(0), traces)
    batch.close()
    ctx.close()
