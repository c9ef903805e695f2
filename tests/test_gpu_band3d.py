"""The 3D band kernel against the FP64 oracle where its y and z slabs take two
nodes of a row per thread (the pair starting at an even column), and on grids
too small for that: rows that end on either half of a pair, with sources and
receivers on both halves, in every slab and beside the Dirichlet columns. Tolerances as in the other forward tests: relative L2 1e-10 in FP64,
1e-4 on traces in FP32."""
import numpy as np
import pytest

import cases


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-10), ("f32", 1e-4)])
@pytest.mark.parametrize("n,halo,freetop", [((25, 22, 23), 6, True), ((180, 152, 131), 30, False),
                                            ((187, 159, 136), 32, True), ((182, 151, 138), 30, False)])
def test_band_pairs_vs_oracle(pkg, oracle, ctx, n, halo, freetop, precision, tol):
    nx, ny, nz = n
    d = 10.0
    rng = np.random.default_rng(nx)
    vel = np.asfortranarray(2000.0 + 500.0 * rng.random(n))
    at = lambda *c: [x * d for x in c]  # noqa: E731  (0-based node)
    src = [at(1, 2, nz // 2), at(2, ny - 3, 3), at(nx - 2, ny // 2, nz - 3), at(nx // 2, 3, nz // 2),
           at(nx // 2 + 1, 3, nz // 2), at(nx // 2, ny // 2, nz // 2)]
    rec = [at(i, j, k) for i in (1, 2, 3, nx // 2, nx - 3, nx - 2) for j in (1, ny // 2, ny - 2)
           for k in (1, halo, nz // 2, nz - 2)]
    lengths = [(m - 1) * d for m in n]
    kw = dict(halo=halo, rcoef=1e-4, freetop=freetop, nt=60)
    t0s = [0.02] * len(src)
    s = pkg.prepare(lengths, None, vel, pkg.Sources(src, t0s, [pkg.rickersource1D] * len(src), 30.0),
                    pkg.Receivers(rec), precision=precision, ppw=1e-9, **kw)
    so = oracle.setup(lengths, None, vel, src, t0s, 30.0, rec, check_ppw=False, dt=s["dt"], **kw)
    field_o, traces_o = oracle.forward(so)
    p = s["problem"]
    traces = np.zeros((p.nt, p.nrec), order="F")
    field = np.zeros(n, order="F")
    ctx.forward(p, s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"], traces, field)
    assert cases.rel_l2(traces, traces_o) <= tol
    if precision == "f64":
        assert cases.rel_l2(field, field_o) <= tol
