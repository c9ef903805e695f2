"""The on-chip loop's bounded wait: a tile that sends no edges makes its neighbours'
waits run out after 2 ms, the run returns AWC_ERR_TIMEOUT and nothing faults; with
the default limit the next run on the same plan gives the exact result. Grids whose
tiles send their edges after the update, before it, and a 1D line."""
import time

import numpy as np
import pytest

import test_gpu_loop2d as loop2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,precision", [((131, 90, 20, True), "f64"), ((409, 333, 20, False), "f32"),
                                            ((1573, 787, 20, True), "f32"), ((1003, 803, 20, True), "f64"),
                                            ((4099, None, 20, False), "f64")])
def test_timeout_and_recovery(pkg, ctx, grid, precision):
    s = loop2d._setup(pkg, grid, precision, seed=1)
    plan = ctx.plan(s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"])
    assert plan.route() == pkg._lib.ROUTE_LOOP
    plan.run()
    traces, field = plan.traces(), plan.field()
    plan.set_wait(rounds=1, round_ns=2000000, withhold=0)
    plan.reset()
    t0 = time.perf_counter()
    with pytest.raises(pkg.AwcError) as ei:
        plan.run()
    assert ei.value.code == pkg._lib.AWC_ERR_TIMEOUT
    assert time.perf_counter() - t0 < 1.0
    plan.set_wait()
    plan.reset()
    plan.run()
    np.testing.assert_array_equal(plan.traces(), traces)
    np.testing.assert_array_equal(plan.field(), field)
    plan.close()


def test_batch_timeout_and_recovery(pkg, ctx):
    setups = [loop2d._setup(pkg, (409, 333, 20, True), "f32", seed=k) for k in (1, 2)]
    p = setups[0]["problem"]
    model = pkg.Problem(ndim=2, precision=p.precision, nx=p.nx, ny=p.ny, nz=1, halo=p.halo,
                        freetop=p.freetop, dx=p.dx, dy=p.dy, dz=1.0, dt=p.dt, nt=p.nt, nsrc=0,
                        nrec=0)
    batch = pkg.Batch(ctx, [model], [setups[0]["vel"]], setups, [0, 0])
    assert batch.launch_count() == 1
    batch.run()
    want = [batch.traces(k) for k in (0, 1)]
    batch.set_wait(rounds=1, round_ns=2000000, withhold=0)
    batch.reset()
    with pytest.raises(pkg.AwcError) as ei:
        batch.run()
    assert ei.value.code == pkg._lib.AWC_ERR_TIMEOUT
    # a failed autotune leaves the launch that was chosen before it
    batch.reset()
    batch.set_launch(16, 4)
    with pytest.raises(pkg.AwcError):
        batch.autotune(8)
    batch.set_wait()
    batch.reset()
    assert batch.get_launch() == (16, 4) and batch.launch_count() == loop2d.NT
    batch.autotune(8)
    assert batch.launch_count() in (1, loop2d.NT)
    batch.run()
    for k in (0, 1):
        np.testing.assert_array_equal(batch.traces(k), want[k])
    batch.close()
