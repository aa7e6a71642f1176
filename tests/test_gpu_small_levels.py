"""The cycle's steps on small levels, run in one launch: more steps than one
launch takes (W-cycles and several sweeps over many levels), the F-cycle, a
base level too large for it, every smoother, partial Dirichlet faces, node
damping, a batch and an algebraic hierarchy -- bit for bit against the oracle
(the tolerance is equality)."""
import numpy as np
import pytest

from _hier import oracle_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gnu_femlisp_b200 as G
    return G


@pytest.fixture(scope="module")
def ctx(G):
    return G.Context(0)


def _cfgs(O, G, smoother, sweeps, gamma, fmg, maxsteps=3):
    C = G._capi
    so = {"jacobi": O.JACOBI, "sor": O.SOR, "ssc": O.SSC, "psc": O.PSC}[smoother]
    sg = {"jacobi": C.FMG_JACOBI, "sor": C.FMG_SOR, "ssc": C.FMG_SSC, "psc": C.FMG_PSC}[smoother]
    damp = {"jacobi": 0.6, "sor": 1.1, "ssc": 1.0, "psc": 0.5}[smoother]
    return (O.solve_cfg(method=O.METHOD_MG, smoother=so, damp=damp, pre=sweeps, post=sweeps, gamma=gamma, compat=False,
                        rtol=1e-12, maxsteps=maxsteps, fmg=fmg),
            G.SolveCfg(C.FMG_METHOD_MG, sg, damp, sweeps, sweeps, gamma, 0, 1.0, 1e-12, 0.0, maxsteps,
                       C.FMG_MULTIPLICATIVE, fmg))


# dim, n0, level, base, Dirichlet mask, smoother, sweeps, gamma, f-cycle, node damping
FORMS = [
    (1, 1, 9, 0, 0b11, "jacobi", 2, 2, 0, False), (1, 3, 6, 0, 0b01, "sor", 3, 1, 1, False),
    (2, 1, 5, 0, 0b1111, "jacobi", 2, 2, 0, True), (2, 1, 6, 0, 0b1111, "jacobi", 1, 1, 1, False),
    (2, 3, 4, 0, 0b0110, "sor", 2, 2, 0, False), (2, 7, 3, 1, 0b1111, "ssc", 1, 1, 0, False),
    (2, 5, 4, 0, 0b1111, "psc", 2, 1, 0, False), (2, 12, 2, 0, 0b1111, "jacobi", 1, 2, 0, False),
    (3, 1, 4, 0, 0b111111, "sor", 1, 2, 0, False), (3, 3, 3, 0, 0b010101, "jacobi", 2, 1, 1, True),
    (3, 5, 2, 0, 0b111111, "ssc", 1, 1, 0, False),
]


@pytest.mark.parametrize("dim,n0,level,base,mask,smoother,sweeps,gamma,fmg,damped", FORMS)
def test_small_levels_bitwise(oracle_mod, G, ctx, dim, n0, level, base, mask, smoother, sweeps, gamma, fmg, damped):
    O, C = oracle_mod, G._capi
    rng = np.random.default_rng(10 * dim + n0)
    o = O.Oracle(dim, 1, level, base_level=base, n0=n0, dirichlet_mask=mask)
    g = G.Grid(ctx, dim, 1, level, base, n0=n0, dirichlet_mask=mask)
    k = np.exp(rng.standard_normal((n0 << level) ** dim))
    o.set_coefficient(O.K_CELL, k)
    g.set_coefficient(C.FMG_K_CELL, k)
    o.assemble()
    g.assemble()
    if damped:
        for l in range(base + 1, level + 1):
            w = rng.uniform(0.45, 0.75, g.nnodes(l))
            o.set_node_damping(l, w)
            g.set_node_damping(l, w)
    oc, gc = _cfgs(O, G, smoother, sweeps, gamma, fmg)
    ref = o.solve(oc)
    x = g.vector()
    hist, steps, _ = g.solve(gc, x)
    assert steps == ref.steps and np.array_equal(hist, ref.history) and np.array_equal(x.get(), ref.x)
    # one cycle on the caller's vectors: its residual too
    b, r = rng.standard_normal(g.nnodes()), None
    X, B, R = g.vector(), g.vector(values=b), g.vector(values=b)
    g.vcycle(gc, X, B, R)
    xo, _, ro = o.vcycle(oc, np.zeros(b.size), b.copy(), b.copy())
    assert np.array_equal(X.get(), xo) and np.array_equal(R.get(), ro)


@pytest.mark.parametrize("smoother,sweeps", [("jacobi", 2), ("sor", 3)])
def test_small_algebraic_levels_bitwise(oracle_mod, G, ctx, smoother, sweeps):
    from gnu_femlisp_b200 import adaptive as AD
    O = oracle_mod
    sizes, mats, interp, rhs = AD.hierarchy(n0=3, levels=4)[:4]
    o = oracle_of(O, sizes, mats, interp, rhs)
    g = G.Grid.algebraic(ctx, sizes)
    for l, m in mats.items():
        g.set_matrix(l, *m)
    for l, m in interp.items():
        g.set_interpolation(l, *m, sizes[l - 1])
    g.set_rhs(rhs)
    oc, gc = _cfgs(O, G, smoother, sweeps, 2, 0)
    ref = o.solve(oc)
    x = g.vector()
    hist, steps, _ = g.solve(gc, x)
    assert steps == ref.steps and np.array_equal(hist, ref.history) and np.array_equal(x.get(), ref.x)


def test_small_levels_of_a_batch(G, ctx):
    """More problems than SMs, whose levels then share an SM: each as by itself."""
    C = G._capi
    cfg = G.SolveCfg(C.FMG_METHOD_CG_MG, C.FMG_JACOBI, 0.6, 1, 1, 1, 0, 1.0, 1e-10, 0.0, 100, C.FMG_MULTIPLICATIVE)
    g = G.Grid(ctx, 2, 1, 5, 0)
    x = g.vector()
    batch = G.Grid.batch(g, 150)
    single = []
    for k in range(150):
        g.set_coefficient(C.FMG_K_CELL, np.exp(np.random.default_rng(k).standard_normal(1024)))
        g.assemble()
        batch.batch_load(k, g)
        if k % 37 == 0:
            x.fill(0.0)
            single.append((k, g.solve(cfg, x)[1], x.get()))
    xb = batch.vector()
    _, steps, _ = batch.batch_solve(cfg, xb)
    xs = xb.get().reshape(150, -1)
    for k, n, xk in single:
        assert steps[k] == n and np.array_equal(xs[k], xk)
