"""The vertex-block substitutions at the ends of the exponent range, where a
quotient by a stored reciprocal does not hold: coefficients and right-hand
sides scaled far up and down, and a last pivot whose reciprocal overflows under
a numerator of zero -- bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gnu_femlisp_b200 as G
    return G


@pytest.fixture(scope="module")
def ctx(G):
    return G.Context(0)


@pytest.mark.parametrize("dim,level", [(1, 4), (2, 3), (3, 2)])
@pytest.mark.parametrize("kscale,bscale", [(1e-250, 1e-50), (1.0, 1e-250), (1e200, 1e250), (1.0, 1.0)])
def test_scaled_sweeps(oracle_mod, G, ctx, dim, level, kscale, bscale):
    O, C = oracle_mod, G._capi
    rng = np.random.default_rng(dim)
    o = O.Oracle(dim, 2, level, base_level=0)
    g = G.Grid(ctx, dim, 2, level, 0)
    k = kscale * np.exp(rng.standard_normal((1 << level) ** dim))
    o.set_coefficient(O.K_CELL, k)
    g.set_coefficient(C.FMG_K_CELL, k)
    o.assemble()
    g.assemble()
    b = bscale * rng.standard_normal(g.nnodes())
    b[::3] = 0.0
    X, B, R = g.vector(), g.vector(values=b), g.vector()
    g.ssc(X, B, R, 1.1)
    xo, ro = o.ssc(np.zeros(b.size), b, np.zeros(b.size), 1.1)
    assert np.isfinite(xo).all() and np.any(xo)
    assert np.array_equal(X.get(), xo) and np.array_equal(R.get(), ro)
    X.fill(0.0)
    g.psc(X, B, 0.7)
    assert np.array_equal(X.get(), o.psc(np.zeros(b.size), b, 0.7))


@pytest.mark.parametrize("pivot", [1e-310, 4e-309, 1e-300])
def test_zero_over_a_tiny_pivot(oracle_mod, G, ctx, pivot):
    # one cell, nodes 0, 1, 2: the block of vertex 0 ends on the pivot itself,
    # that of vertex 2 takes node 2's row first
    O = oracle_mod
    A = np.array([[1.0, 0.0, 0.0], [0.0, pivot, 1.0], [0.0, 1.0, 1.0]])
    slots = np.zeros((5, 3))
    for i in range(3):
        for j in range(3):
            slots[j - i + 2, i] = A[i, j]
    b = np.array([1.0, 0.0, 0.0])
    o = O.Oracle(1, 2, 0, dirichlet_mask=0).set_levels({0: slots}, b)
    g = G.Grid(ctx, 1, 2, 0, 0, dirichlet_mask=0)
    i, j = np.nonzero(A)
    g.set_matrix(0, np.searchsorted(i, np.arange(4)), j, A[i, j])
    X, B, R = g.vector(), g.vector(values=b), g.vector()
    g.ssc(X, B, R, 1.0)
    xo, ro = o.ssc(np.zeros(3), b, np.zeros(3), 1.0)
    assert np.isfinite(xo).all()
    assert np.array_equal(X.get(), xo) and np.array_equal(R.get(), ro)
