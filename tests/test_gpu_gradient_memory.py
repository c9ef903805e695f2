"""Device memory of the gradients: the run's fields are kept whole only where that
leaves room, what the outputs need is had first, the caller's limit holds, and a
plan or batch without room gets the memory that the gradients hold. Most of the
device is filled by one allocation that nothing touches."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, NT, EVERY = (200, 190, 180), 40, 8


def _setup(pkg, nt=NT, n=N):
    rng = np.random.default_rng(5)
    vel = np.asfortranarray(2000.0 + 200.0 * rng.random(n))
    srcs = pkg.Sources([[m * 5.0 for m in n]], [0.02], [pkg.rickersource1D], 30.0)
    s = pkg.prepare([(m - 1) * 10.0 for m in n], None, vel, srcs,
                    pkg.Receivers([[m * 5.0 + 30.0 for m in n]]), halo=6, ppw=1e-9, precision="f64", nt=nt)
    return s, np.zeros((nt, 1))


def _free():
    return torch.cuda.mem_get_info()[0]


def _fill(leave):
    """Holds all but about `leave` bytes of the device."""
    torch.cuda.empty_cache()
    return torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")


def test_room_for_everything_else(pkg):
    """The device has room for the whole run's fields but not for the output as
    well: the run keeps to its segments, as it did where it had to before."""
    s, obs = _setup(pkg)
    for _ in range(2):  # the first one loads the kernels
        ctx = pkg.Context(0)
        ctx.set_autotune(0)
        before = _free()
        want = pkg.adjoint.misfit_gradient(s, obs, EVERY, ctx)
        used = before - _free()
        assert ctx.last_segments() == 1 and np.abs(want[1]).max() > 0.0
        ctx.close()
    hold = _fill(used - np.prod(N) * 8 // 2)
    ctx = pkg.Context(0)
    ctx.set_autotune(0)
    for _ in range(2):
        got = pkg.adjoint.misfit_gradient(s, obs, EVERY, ctx)
        assert ctx.last_segments() == NT // EVERY
        assert got[0] == want[0]
        np.testing.assert_array_equal(got[1], want[1])
    ctx.close()
    del hold
    torch.cuda.empty_cache()


def test_limit(pkg):
    s, obs = _setup(pkg)
    ctx = pkg.Context(0)
    ctx.set_autotune(0)
    before = _free()
    ctx.set_keep_limit(0)
    a = pkg.adjoint.misfit_gradient(s, obs, EVERY, ctx)
    assert ctx.last_segments() == NT // EVERY
    parts = before - _free()
    ctx.set_keep_limit(-1)
    b = pkg.adjoint.misfit_gradient(s, obs, EVERY, ctx)
    assert ctx.last_segments() == 1 and before - _free() > parts
    np.testing.assert_array_equal(a[1], b[1])
    ctx.close()


def test_plans_and_batches_get_the_memory_back(pkg):
    """A gradient's arena held between calls makes way for a plan and for a batch
    that the device has no room for beside it."""
    s, obs = _setup(pkg)
    ctx = pkg.Context(0)
    ctx.set_autotune(0)
    s2, _ = _setup(pkg, nt=4, n=(230, 220, 210))  # 0.6 GB: less than the arena
    model = pkg.Problem(ndim=2, precision=pkg.AWC_F64, nx=4000, ny=3000, nz=1, halo=6, freetop=1,
                        dx=10.0, dy=10.0, dz=1.0, dt=1e-3, nt=4, nsrc=0, nrec=0)
    vel2 = np.full((4000, 3000), 2000.0, order="F")
    shot = pkg.prepare([39990.0, 29990.0], None, vel2,
                       pkg.Sources([[500.0, 500.0]], [0.02], [pkg.rickersource1D], 30.0),
                       pkg.Receivers([[500.0, 300.0]]), halo=6, ppw=1e-9, precision="f64", nt=4)
    for make in (lambda: ctx.plan(s2["problem"], s2["vel"], s2["coeffs"], s2["possrcs"],
                                  s2["dt2srctf"], s2["posrecs"]),
                 lambda: pkg.Batch(ctx, [model], [vel2], [shot], [0])):
        pkg.adjoint.misfit_gradient(s, obs, EVERY, ctx)
        assert ctx.last_segments() == 1
        hold = _fill(64 << 20)
        made = make()
        made.run()
        made.close()
        del hold
        torch.cuda.empty_cache()
    ctx.close()


def test_single_and_multi_shot_calls_share_their_memory(pkg):
    s, obs = _setup(pkg)
    ctx = pkg.Context(0)
    ctx.set_autotune(0)
    J, grad = pkg.adjoint.misfit_gradient_shots([s], [obs], EVERY, ctx)
    free = _free()
    for _ in range(2):
        one = pkg.adjoint.misfit_gradient(s, obs, EVERY, ctx)
        assert _free() == free and one[0] == J
        np.testing.assert_array_equal(one[1], grad)
        pkg.adjoint.misfit_gradient_shots([s], [obs], EVERY, ctx)
        assert _free() == free
    ctx.close()
