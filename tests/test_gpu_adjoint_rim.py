"""adjoint_sources of a source on the Dirichlet rim: no adjoint, so zero, whatever
the context's working memory held before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n", [(40, 30), (24, 20, 22)])
def test_rim_sources_are_zero(pkg, n, precision):
    ctx, nt = pkg.Context(0), 50
    inside = [5 * 10.0] * len(n)

    def setup(first):
        srcs = pkg.Sources([first, [60.0] * len(n)], [0.02] * 2, [pkg.rickersource1D] * 2, 30.0)
        return pkg.prepare([(m - 1) * 10.0 for m in n], None, np.full(n, 2000.0, order="F"), srcs,
                           pkg.Receivers([[80.0] * len(n)]), halo=4, ppw=1e-9, precision=precision,
                           nt=nt)

    r = np.asfortranarray(np.random.default_rng(4).standard_normal((nt, 1)))
    a = pkg.adjoint.adjoint_sources(setup(inside), r, ctx)
    assert np.abs(a[:, 0]).max() > 0.0  # now in the memory that the next call gets
    b = pkg.adjoint.adjoint_sources(setup([0.0] + inside[1:]), r, ctx)
    np.testing.assert_array_equal(b[:, 0], 0.0)
    np.testing.assert_array_equal(b[:, 1], a[:, 1])
    ctx.close()
