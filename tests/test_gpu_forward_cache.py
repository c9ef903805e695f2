"""awc_forward's plan cache: 1D lines do not push 2D and 3D plans out of it (nor
the other way round), and of each the two most recent shapes stay."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _forward(pkg, ctx, n, nt=12):
    srcs = pkg.Sources([[m * 5.0 for m in n]], [0.02], [pkg.rickersource1D], 30.0)
    s = pkg.prepare([(m - 1) * 10.0 for m in n], None, np.full(n, 2000.0, order="F"), srcs,
                    pkg.Receivers([[m * 5.0 + 10.0 for m in n]]), halo=5, ppw=1e-9, nt=nt)
    traces = np.zeros((nt, 1), order="F")
    ctx.forward(s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"], s["posrecs"],
                traces)
    return traces


def test_lines_and_grids_have_their_own_places(pkg):
    ctx = pkg.Context(0)
    grids = [(1500, 1400), (150, 140, 130)]  # 16 and 22 MB a field
    first = [_forward(pkg, ctx, n) for n in grids]
    free = torch.cuda.mem_get_info()[0]
    lines = [_forward(pkg, ctx, (n,)) for n in (301, 401, 501)]
    # the grids' plans are still there: their memory was not given back
    assert torch.cuda.mem_get_info()[0] <= free + (8 << 20)
    for n, want in zip(grids, first):
        np.testing.assert_array_equal(_forward(pkg, ctx, n), want)
    np.testing.assert_array_equal(_forward(pkg, ctx, (301,)), lines[0])
    # a third grid takes the place of the oldest
    free = torch.cuda.mem_get_info()[0]
    _forward(pkg, ctx, (100, 90))
    assert torch.cuda.mem_get_info()[0] >= free + (32 << 20)
    ctx.close()
