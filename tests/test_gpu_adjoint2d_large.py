"""2D adjoint steps of grids of several waves of blocks, whose blocks outside the
bands take the body without band terms; zone edges on, before and after a block's
edge. Dot-product test (FP64, 1e-12 as in test_gpu_adjoint.py), the gradient along
a random direction against central differences of the forward run (FP64, 1e-6 as
there), and FP32 against FP64 (relative L2 1e-4 as there)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

GRIDS = [(702, 600, 20, True), (1030, 421, 31, False), (515, 1203, 30, True), (901, 466, 6, False)]


def _setup(pkg, grid, precision, nt=110):
    nx, ny, halo, freetop = grid
    rng = np.random.default_rng(nx)
    d = 10.0
    vel = np.asfortranarray(2000.0 + 300.0 * rng.random((nx, ny)))
    src = [[(nx // 2) * d, 9 * d], [(halo // 2) * d, (ny // 2) * d], [(nx - 5) * d, (ny - 4) * d]]
    rec = [[i * d, j * d] for i in range(2, nx - 2, 97) for j in (3, halo + 2, ny // 2, ny - 3)]
    return pkg.prepare([(nx - 1) * d, (ny - 1) * d], None, vel,
                       pkg.Sources(src, [0.03] * 3, [pkg.rickersource1D] * 3, 25.0),
                       pkg.Receivers(rec), halo=halo, freetop=freetop, ppw=1e-9,
                       precision=precision, nt=nt)


def _traces(ctx, s):
    p = s["problem"]
    tr = np.zeros((p.nt, p.nrec), order="F")
    ctx.forward(p, s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"], tr)
    return tr


@pytest.mark.parametrize("grid", GRIDS)
def test_dot_product(pkg, ctx, grid):
    s = _setup(pkg, grid, "f64")
    p = s["problem"]
    rng = np.random.default_rng(1)
    q = np.asfortranarray(rng.standard_normal((p.nt, p.nsrc)))
    r = np.asfortranarray(rng.standard_normal((p.nt, p.nrec)))
    traces = _traces(ctx, dict(s, dt2srctf=q))
    lhs = float((traces * r).sum())
    rhs = float((q * pkg.adjoint.adjoint_sources(s, r, ctx)).sum())
    scale = np.linalg.norm(traces) * np.linalg.norm(r)
    assert abs(lhs) > 1e-6 * scale
    assert abs(lhs - rhs) <= 1e-12 * scale


@pytest.mark.parametrize("grid", GRIDS)
def test_gradient_along_a_direction(pkg, ctx, grid):
    s = _setup(pkg, grid, "f64")
    p = s["problem"]
    _, grad, _ = pkg.adjoint.misfit_gradient(s, np.zeros((p.nt, p.nrec)), 50, ctx)
    c2, w = s["vel"] ** 2, np.random.default_rng(2).standard_normal(s["vel"].shape)
    w[:, 0] = w[:, -1] = w[0, :] = w[-1, :] = 0.0  # the rim's velocity has no effect
    eps = 1e-4

    def misfit(e):
        vel = np.asfortranarray(np.sqrt(c2 * (1.0 + e * w)))
        return 0.5 * float((_traces(ctx, dict(s, vel=vel)) ** 2).sum())

    diff = (misfit(eps) - misfit(-eps)) / (2.0 * eps)
    assert abs(float((grad * c2 * w).sum()) - diff) <= 1e-6 * abs(diff)
    s32 = _setup(pkg, grid, "f32")
    _, grad32, _ = pkg.adjoint.misfit_gradient(s32, np.zeros((p.nt, p.nrec)), 50, ctx)
    assert cases.rel_l2(grad32, grad) <= 1e-4
