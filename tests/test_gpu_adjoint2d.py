"""The one-launch 2D adjoint step: dot-product test (FP64, 1e-12 as in
test_gpu_adjoint.py) with receivers and sources that share nodes, repeat, lie in
the CPML bands and on the Dirichlet rim, at sizes around a block's 32 x 8 nodes;
and segments (recomputed fields) against one segment, bitwise, on a run whose
fields are too large to be kept whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(pkg, nx, ny, halo, freetop, nt, nsrc=7, nrec=40, precision="f64"):
    rng = np.random.default_rng(nx + ny)
    d = 10.0
    vel = np.asfortranarray(2000.0 + 800.0 * rng.random((nx, ny)))

    def nodes(k):
        p = np.stack([rng.integers(0, nx, k), rng.integers(0, ny, k)], axis=1)
        p[-1], p[0] = p[1], (min(2, nx - 2), ny // 2)  # a repeat, a band node
        return p

    src, rec = nodes(nsrc), nodes(nrec)
    rec[2] = src[0]  # a receiver on a source node
    srcs = pkg.Sources((src * d).tolist(), [0.02] * nsrc, [pkg.rickersource1D] * nsrc, 30.0)
    return pkg.prepare([(nx - 1) * d, (ny - 1) * d], None, vel, srcs,
                       pkg.Receivers((rec * d).tolist()), halo=halo, freetop=freetop, ppw=1e-9,
                       precision=precision, nt=nt)


@pytest.mark.parametrize("nx,ny,halo,freetop", [(18, 18, 8, False), (34, 10, 4, True),
                                                (35, 11, 3, False), (66, 43, 20, False),
                                                (97, 64, 10, True)])
def test_dot_product(pkg, ctx, nx, ny, halo, freetop):
    s = _setup(pkg, nx, ny, halo, freetop, nt=90)
    p = s["problem"]
    rng = np.random.default_rng(1)
    q = np.asfortranarray(rng.standard_normal((p.nt, p.nsrc)))
    rim = ((s["possrcs"] == 1) | (s["possrcs"] == np.array([nx, ny]))).any(axis=1)
    rim_r = ((s["posrecs"] == 1) | (s["posrecs"] == np.array([nx, ny]))).any(axis=1)
    q[:, rim] = 0.0  # rim nodes have no adjoint
    r = np.asfortranarray(rng.standard_normal((p.nt, p.nrec)))
    r[:, rim_r] = 0.0
    traces = np.zeros((p.nt, p.nrec), order="F")
    ctx.forward(p, s["vel"], s["coeffs"], s["possrcs"], q, s["posrecs"], traces)
    a = pkg.adjoint.adjoint_sources(s, r, ctx)
    lhs, rhs = float((traces * r).sum()), float((q[:, ~rim] * a[:, ~rim]).sum())
    scale = np.linalg.norm(traces) * np.linalg.norm(r)
    assert abs(lhs) > 1e-6 * scale
    assert abs(lhs - rhs) <= 1e-12 * scale


def test_segments_equal_one_segment(pkg, ctx):
    s = _setup(pkg, 1101, 1003, 20, True, nt=150)  # 152 fields of 9 MB: more than are kept whole
    obs = np.asfortranarray(np.random.default_rng(2).standard_normal((150, s["problem"].nrec))) * 1e-9
    whole = pkg.adjoint.misfit_gradient(s, obs, 150, ctx)
    parts = pkg.adjoint.misfit_gradient(s, obs, 40, ctx)
    assert whole[0] == parts[0] and np.abs(whole[1]).max() > 0.0
    np.testing.assert_array_equal(parts[1], whole[1])
    np.testing.assert_array_equal(parts[2], whole[2])
