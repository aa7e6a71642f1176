"""An SOR sweep of a Q1 level that is given one vector as solution and as
residual (not refused): every row adds to what it has just written, as the
oracle's rows do on one array -- bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n0,level", [(1, 3, 4), (2, 5, 3), (3, 1, 3)])
def test_sor_with_one_vector(oracle_mod, dim, n0, level):
    import gnu_femlisp_b200 as G
    O, ctx = oracle_mod, G.Context(0)
    k = np.exp(np.random.default_rng(dim).standard_normal((n0 << level) ** dim))
    o = O.Oracle(dim, 1, level, n0=n0)
    g = G.Grid(ctx, dim, 1, level, 0, n0=n0)
    o.set_coefficient(O.K_CELL, k)
    g.set_coefficient(G._capi.FMG_K_CELL, k)
    o.assemble()
    g.assemble()
    rng = np.random.default_rng(level)
    x, b = rng.standard_normal(g.nnodes()), rng.standard_normal(g.nnodes())
    X = g.vector(values=x)
    g.sor(X, g.vector(values=b), X, 1.1)
    O.lib().ora_sor(o.h, level, 1.1, O._p(x), O._p(b), O._p(x))
    assert np.array_equal(X.get(), x)
