"""The on-chip 2D time loop (runs of eight steps or more on grids that fit the
chip) against the per-step kernels (shorter runs): the same arithmetic in the
same order, so every output is bitwise the same, whatever the tiling. Sizes:
one node wide interiors, a tile's vector width and its remainders, one tile,
several tiles in one and both directions, more receivers than threads, bands
that meet, per-step grids of one node per thread and of strips (the largest), sources on the Dirichlet rim and on tile edges."""
import numpy as np
import pytest

NT = 60

# (nx, ny, halo, free top): ny = None is a 1D line
GRIDS = [(3, 3, 0, False), (4, 5, 1, False), (5, 4, 1, True), (23, 19, 8, False),
         (43, 42, 20, False), (64, 67, 5, True), (131, 90, 20, True), (257, 61, 10, False),
         (70, 401, 20, True), (409, 333, 20, False), (1030, 517, 30, True),
         (1039, 1037, 20, False), (2083, 1019, 20, True), (3, None, 0, False),
         (129, None, 20, False), (4099, None, 20, False)]


def _setup(pkg, grid, precision, seed):
    nx, ny, halo, freetop = grid
    rng = np.random.default_rng(seed)
    shape = (nx,) if ny is None else (nx, ny)
    d = 10.0
    vel = 1500.0 + 1000.0 * rng.random(shape)
    lengths = [(n - 1) * d for n in shape]

    def nodes(k):  # anywhere, rim and corners included, some twice
        p = np.stack([rng.integers(0, n, k) for n in shape], axis=1) * d
        p[-1] = p[0]
        return p.tolist()

    src = nodes(9)
    srcs = pkg.Sources(src, [0.02] * 9, [pkg.rickersource1D] * 9, 30.0)
    recs = pkg.Receivers(nodes(700))
    return pkg.prepare(lengths, None, vel, srcs, recs, halo=halo, freetop=freetop,
                       precision=precision, ppw=0.1, nt=NT)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(str(v) for v in g))
def test_loop_equals_per_step_kernels(pkg, grid, precision):
    ctx = pkg.default_context(0)
    s = _setup(pkg, grid, precision, seed=grid[0])
    args = (s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"])
    plan = ctx.plan(*args)
    while plan.step < NT:
        plan.run(7)  # too short for the loop
    traces, field = plan.traces(), plan.field()
    assert np.abs(traces).max() > 0.0
    plan.reset()
    plan.run()
    np.testing.assert_array_equal(plan.traces(), traces)
    np.testing.assert_array_equal(plan.field(), field)
    # loop and per-step runs hand the whole state to one another
    plan.reset()
    for n in (8, 3, 17, 1, 25, 2, NT):
        plan.run(n)
    np.testing.assert_array_equal(plan.traces(), traces)
    np.testing.assert_array_equal(plan.field(), field)
    plan.close()
