"""The tests that compare one route with another are worth what they run: here
the grids of test_gpu_loop2d, test_gpu_band3d and the gradient tests are held to
the route they stand for. And the strip kernel, whose grids the loop cannot take,
against the batch's step kernels: the same bits."""
import numpy as np
import pytest

import test_gpu_loop2d as loop2d

pytestmark = pytest.mark.gpu


LARGE = {(1039, "f64"), (2083, "f32"), (2083, "f64")}  # fields of 8 MB and more


def _args(s):
    return s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("grid", loop2d.GRIDS, ids=lambda g: "x".join(str(v) for v in g))
def test_loop_grids_take_the_loop(pkg, ctx, grid, precision):
    nx, ny, halo, freetop = grid
    plan = ctx.plan(*_args(loop2d._setup(pkg, grid, precision, seed=nx)))
    step = pkg._lib.ROUTE_STRIPS if (nx, precision) in LARGE else 0
    # two bands of an axis that share a face, or too large a grid: step by step
    meet = halo > 0 and (nx <= 2 * halo + 2 or (ny is not None and not freetop and ny <= 2 * halo + 2))
    loop = not meet and (nx, precision) not in (LARGE - {(2083, "f32")})
    assert plan.route() == (pkg._lib.ROUTE_LOOP if loop else step)
    assert plan.launch_count() == (1 if loop else loop2d.NT)
    assert plan.route(7) == step and plan.launch_count(7) == 7
    plan.close()


@pytest.mark.parametrize("grid", [(1003, 803, 20, True), (871, 859, 30, False)])
def test_loop_equals_per_step_kernels_f64(pkg, ctx, grid):
    """Grids near the most that fit in FP64 (those of test_gpu_loop2d run step by step)."""
    plan = ctx.plan(*_args(loop2d._setup(pkg, grid, "f64", seed=grid[0])))
    assert plan.route() == pkg._lib.ROUTE_LOOP
    plan.close()
    loop2d.test_loop_equals_per_step_kernels(pkg, grid, "f64")


@pytest.mark.parametrize("grid,precision", [((2083, 1019, 20, True), "f64"),
                                            ((2498, 1203, 9, False), "f64"),
                                            ((3073, 1601, 20, True), "f32"),
                                            ((2690, 1807, 0, False), "f32")])
def test_strips_equal_batch_kernels(pkg, ctx, grid, precision):
    _equals_batch(pkg, ctx, grid, precision, pkg._lib.ROUTE_STRIPS)


def _equals_batch(pkg, ctx, grid, precision, route):
    s = loop2d._setup(pkg, grid, precision, seed=grid[0])
    p = s["problem"]
    plan = ctx.plan(*_args(s))
    assert plan.route() == route
    plan.run()
    model = pkg.Problem(ndim=2, precision=p.precision, nx=p.nx, ny=p.ny, nz=1, halo=p.halo,
                        freetop=p.freetop, dx=p.dx, dy=p.dy, dz=1.0, dt=p.dt, nt=p.nt, nsrc=0,
                        nrec=0)
    batch = pkg.Batch(ctx, [model], [s["vel"]], [s], [0])
    batch.set_launch(8, 8)
    batch.run()
    assert np.abs(plan.traces()).max() > 0.0
    np.testing.assert_array_equal(plan.traces(), batch.traces(0))
    np.testing.assert_array_equal(plan.field(), batch.field(0))
    batch.close()
    plan.close()


@pytest.mark.parametrize("grid,precision", [((130, 19000, 10, True), "f32"),
                                            ((260, 9500, 4, True), "f32"),
                                            ((70, 20000, 18, False), "f64")])
def test_narrow_grids_take_one_node_per_thread(pkg, ctx, grid, precision):
    """Beyond the chip, but of few strips a row, most of them in the x bands: strips
    take up to twice the time there. The same bits as the batch's step kernels."""
    _equals_batch(pkg, ctx, grid, precision, 0)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n,halo,freetop,pairs",
                         [((25, 22, 23), 6, True, False), ((180, 152, 131), 30, False, True),
                          ((187, 159, 136), 32, True, True), ((182, 151, 138), 30, False, True)])
def test_band_grids_take_pairs(pkg, ctx, n, halo, freetop, pairs, precision):
    srcs = pkg.Sources([[m * 5.0 for m in n]], [0.02], [pkg.rickersource1D], 30.0)
    s = pkg.prepare([(m - 1) * 10.0 for m in n], None, np.full(n, 2000.0), srcs,
                    pkg.Receivers([[20.0] * 3]), halo=halo, freetop=freetop, precision=precision,
                    ppw=1e-9, nt=2)
    plan = ctx.plan(*_args(s))
    assert plan.route() == (pkg._lib.ROUTE_BAND_PAIRS if pairs else 0)
    plan.close()


@pytest.mark.parametrize("n,halo,nt,segments", [((1101, 1003), 20, 150, {150: 1, 40: 4}),
                                                ((120, 110, 115), 12, 100, {100: 1, 34: 1, 20: 5})])
def test_gradient_segments(pkg, ctx, n, halo, nt, segments):
    srcs = pkg.Sources([[m * 5.0 for m in n]], [0.02], [pkg.rickersource1D], 30.0)
    s = pkg.prepare([(m - 1) * 10.0 for m in n], None, np.full(n, 2000.0), srcs,
                    pkg.Receivers([[200.0] * len(n)]), halo=halo, ppw=1e-9, precision="f64", nt=nt)
    for every, want in segments.items():
        pkg.adjoint.misfit_gradient(s, np.zeros((nt, 1)), every, ctx)
        assert ctx.last_segments() == want
