"""The level operators at the sizes where a row kernel can go wrong -- a block
partly filled, one node more than a block, ragged root sizes, one or two cells
a side, Dirichlet conditions on some faces only -- bit for bit against the
oracle (the tolerance is equality: both sides fix one operation order)."""
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


# dim, order, components, n0, level, Dirichlet mask
FORMS = [
    (1, 1, 1, 127, 1, 0b11), (1, 1, 1, 64, 1, 0b01), (1, 2, 1, 5, 3, 0b10), (2, 1, 1, 3, 3, 0b1111),
    (2, 1, 1, 7, 2, 0b0110), (2, 2, 1, 1, 1, 0b1111), (2, 2, 1, 3, 3, 0b0001), (3, 1, 1, 1, 1, 0b111111),
    (3, 1, 1, 5, 2, 0b111111), (3, 1, 1, 3, 2, 0b010110), (3, 2, 1, 1, 1, 0b111111), (3, 2, 1, 3, 2, 0b111111),
    (3, 2, 1, 2, 2, 0b000001), (3, 2, 3, 1, 1, 0b000001), (3, 2, 3, 3, 1, 0b000001), (3, 2, 3, 2, 2, 0b011001),
    (3, 1, 3, 3, 2, 0b000001),
]


@pytest.mark.parametrize("dim,order,nc,n0,level,mask", FORMS)
def test_operators_bitwise(oracle_mod, G, ctx, dim, order, nc, n0, level, mask):
    C, O = G._capi, oracle_mod
    rng = np.random.default_rng(100 * dim + n0)
    o = O.Oracle(dim, order, level, base_level=0, ncomp=nc, n0=n0, dirichlet_mask=mask)
    g = G.Grid(ctx, dim, order, level, 0, n0=n0, ncomp=nc, dirichlet_mask=mask)
    k = np.exp(rng.standard_normal((n0 << level) ** dim))
    o.set_coefficient(O.K_CELL if nc == 1 else O.LAMBDA_MU_CELL, k)
    g.set_coefficient(C.FMG_K_CELL if nc == 1 else C.FMG_LAMBDA_MU_CELL, k)
    o.assemble()
    g.assemble()
    for l in range(level + 1):
        n = g.nnodes(l) * nc
        x, b = rng.standard_normal(n), rng.standard_normal(n)
        X, B, Y = g.vector(l, x), g.vector(l, b), g.vector(l)
        g.matvec(X, Y)
        assert np.array_equal(Y.get(), o.matvec(x, l)), f"matvec {l}"
        g.residual(X, B, Y)
        assert np.array_equal(Y.get(), o.residual(x, b, l)), f"residual {l}"
        if l == 0:
            g.coarse_solve(X, B, 0.9)
            xo, ro = o.coarse_solve(x, b, 0.9)
            assert np.array_equal(X.get(), xo) and np.array_equal(B.get(), ro), "coarse solve"
            continue
        g.jacobi(X, B, 0.6)
        xo, ro = o.jacobi(x, b, 0.6, l)
        assert np.array_equal(X.get(), xo) and np.array_equal(B.get(), ro), f"jacobi {l}"
        if nc == 1:
            for sweep, ref in ((g.sor, o.sor), (g.ssc, o.ssc)):
                X.set(x), B.set(b), Y.fill(0.0)
                sweep(X, B, Y, 1.1)
                xo, ro = ref(x, b, np.zeros(n), 1.1, l)
                assert np.array_equal(X.get(), xo) and np.array_equal(Y.get(), ro), f"{ref.__name__} {l}"
        X.set(x)
        rc = g.vector(l - 1)
        g.restrict(X, rc)
        assert np.array_equal(rc.get(), o.restrict(x, l)), f"restrict {l}"
        xc = rng.standard_normal(g.nnodes(l - 1) * nc)
        g.prolongate(g.vector(l - 1, xc), B.set(b))
        assert np.array_equal(B.get(), o.prolongate(xc, b, l - 1)), f"prolongate {l}"
