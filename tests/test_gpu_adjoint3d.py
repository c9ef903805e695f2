"""The 3D adjoint step's shell in node pairs, and its sources and residuals in
one launch: dot-product test (FP64, 1e-12 as in test_gpu_adjoint.py) at odd and
even row lengths, with grids whose x bands' zones leave one node, two nodes or a
core between them, on sources and receivers that share nodes, repeat, lie in the
bands and on the Dirichlet rim; and segments against runs whose fields are kept."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,halo,freetop", [((13, 17, 18), 4, False), ((14, 18, 17), 4, True),
                                            ((15, 40, 21), 4, False), ((39, 22, 36), 6, True),
                                            ((74, 31, 29), 5, False)])
def test_dot_product(pkg, ctx, n, halo, freetop):
    rng = np.random.default_rng(sum(n))
    d, nt, nn = 10.0, 70, np.array(n)
    vel = np.asfortranarray(2000.0 + 800.0 * rng.random(n))

    def nodes(k):
        p = np.stack([rng.integers(0, m, k) for m in n], axis=1)
        p[-1], p[0] = p[1], (n[0] // 2, min(2, n[1] - 2), n[2] // 2)  # a repeat, a band node
        return p

    src, rec = nodes(7), nodes(150)
    rec[2] = src[0]  # a receiver on a source node
    srcs = pkg.Sources((src * d).tolist(), [0.02] * 7, [pkg.rickersource1D] * 7, 30.0)
    s = pkg.prepare(((nn - 1) * d).tolist(), None, vel, srcs, pkg.Receivers((rec * d).tolist()),
                    halo=halo, freetop=freetop, ppw=1e-9, precision="f64", nt=nt)
    p = s["problem"]
    rim = ((s["possrcs"] == 1) | (s["possrcs"] == nn)).any(axis=1)
    rim_r = ((s["posrecs"] == 1) | (s["posrecs"] == nn)).any(axis=1)
    q = np.asfortranarray(rng.standard_normal((p.nt, p.nsrc)))
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
    """100 fields of 12 MB: kept whole for intervals of 100 and 34 steps, by
    segments for 20; the same bits."""
    n, nt = (120, 110, 115), 100
    rng = np.random.default_rng(3)
    vel = np.asfortranarray(2000.0 + 800.0 * rng.random(n))
    pos = [[300.0, 400.0, 300.0], [700.0, 20.0, 600.0]]
    srcs = pkg.Sources(pos[:1], [0.02], [pkg.rickersource1D], 30.0)
    s = pkg.prepare([(m - 1) * 10.0 for m in n], None, vel, srcs, pkg.Receivers(pos), halo=12,
                    ppw=1e-9, precision="f64", nt=nt)
    obs = np.asfortranarray(rng.standard_normal((nt, 2))) * 1e-9
    want = pkg.adjoint.misfit_gradient(s, obs, nt, ctx)
    assert np.abs(want[1]).max() > 0.0
    for every in (34, 20):
        got = pkg.adjoint.misfit_gradient(s, obs, every, ctx)
        assert got[0] == want[0]
        np.testing.assert_array_equal(got[1], want[1])
        np.testing.assert_array_equal(got[2], want[2])
