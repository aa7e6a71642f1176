"""The kernels that large levels take, on levels just above the sizes where
they take over and just below: the FP64 ones and the matrix-free operator bit
for bit against the oracle, and the FP32 cycles of the mixed solves through
its first step against the same step with the FP64 cycle.

Bounds of the latter, from the unit roundoffs 2^-24 (FP32) and 2^-9 (BF16):
- vector form: a row sum of m terms is off by m 2^-24 of its terms' size; the
  five row sums a level of V(2,2) and the transfers, on every level, give
  8 m 2^-24 per level;
- scalar form: the coarse right-hand sides and residuals are BF16, two
  roundings a level of 2^-9 of that level's correction each."""
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


def make_pair(O, G, ctx, order, nc, n0, level, mask, assemble=True):
    o = O.Oracle(3, order, level, base_level=0, ncomp=nc, n0=n0, dirichlet_mask=mask)
    g = G.Grid(ctx, 3, order, level, 0, n0=n0, ncomp=nc, dirichlet_mask=mask)
    k = np.exp(0.5 * np.random.default_rng(n0 + level).standard_normal((n0 << level) ** 3))
    g.set_coefficient(G._capi.FMG_K_CELL if nc == 1 else G._capi.FMG_LAMBDA_MU_CELL, k)
    g.assemble()
    if assemble:
        o.set_coefficient(O.K_CELL if nc == 1 else O.LAMBDA_MU_CELL, k)
        o.assemble()
    return o, g


# nodes a side 33, 49, 65, 97: the SSC's residuals by tiles up to 33, the SOR's colours up to 65
@pytest.mark.parametrize("n0,level,mask", [(1, 4, 0b111111), (3, 3, 0b011001), (1, 5, 0b000100), (3, 4, 0b111111)])
def test_q2_sweeps(oracle_mod, G, ctx, n0, level, mask):
    o, g = make_pair(oracle_mod, G, ctx, 2, 1, n0, level, mask)
    rng = np.random.default_rng(level)
    n = g.nnodes()
    x, b, r = (rng.standard_normal(n) for _ in range(3))
    for sweep, ref in ((g.sor, o.sor), (g.ssc, o.ssc)):
        X, B, R = g.vector(values=x), g.vector(values=b), g.vector(values=r)
        sweep(X, B, R, 1.1)
        xo, ro = ref(x, b, r, 1.1)
        assert np.array_equal(X.get(), xo) and np.array_equal(R.get(), ro), ref.__name__
    Y = g.vector()
    g.residual(g.vector(values=x), g.vector(values=b), Y)
    assert np.array_equal(Y.get(), o.residual(x, b))


# Q2 by threads per scalar unknown and, from 33^3 coarse and 49^3 fine nodes on, per node; Q1 per unknown
@pytest.mark.parametrize("order,n0,level", [(2, 3, 3), (2, 1, 5), (1, 7, 3), (1, 1, 6)])
def test_vector_transfers(oracle_mod, G, ctx, order, n0, level):
    o, g = make_pair(oracle_mod, G, ctx, order, 3, n0, level, 0b011001, assemble=False)
    rng = np.random.default_rng(level)
    for l in range(1, level + 1):
        x, xc = rng.standard_normal(3 * g.nnodes(l)), rng.standard_normal(3 * g.nnodes(l - 1))
        X, XC = g.vector(l, x), g.vector(l - 1)
        g.restrict(X, XC)
        assert np.array_equal(XC.get(), o.restrict(x, l)), f"restrict {l}"
        g.prolongate(XC.set(xc), X)
        assert np.array_equal(X.get(), o.prolongate(xc, x, l - 1)), f"prolongate {l}"


# nodes a side 21 to 41 (Q1), 17 to 49 (Q2): FP32 rows a thread per scalar row below 12,000 nodes, per node above
@pytest.mark.parametrize("order,n0,level", [(1, 5, 2), (1, 3, 3), (1, 7, 2), (1, 5, 3), (2, 1, 3), (2, 3, 2), (2, 1, 4), (2, 3, 3)])
def test_mixed_vector_step(oracle_mod, G, ctx, order, n0, level):
    O, C = oracle_mod, G._capi
    o, g = make_pair(O, G, ctx, order, 3, n0, level, 0b000001)
    m = round(g.nnodes() ** (1 / 3))
    b = np.random.default_rng(1).standard_normal((g.nnodes(), 3))
    b[np.arange(g.nnodes()) % m == 0] = 0.0
    b = b.reshape(-1)
    g.set_rhs(b)
    oc = O.solve_cfg(method=O.METHOD_MG, smoother=O.JACOBI, damp=0.6, pre=2, post=2, compat=False)
    z, _, _ = o.vcycle(oc, np.zeros(b.size), b, b)
    want = (z @ b) / (z @ o.matvec(z)) * z
    X = g.vector()
    g.solve_mixed(G.SolveCfg(C.FMG_METHOD_CG_MG, C.FMG_JACOBI, 0.6, 2, 2, 1, 0, 1.0, 1e-30, 0.0, 0,
                             C.FMG_MULTIPLICATIVE), X)
    terms = 3 * (2 * order + 1) ** 3
    diff = np.max(np.abs(X.get() - want)) / np.max(np.abs(want))
    print("relative difference", diff)
    assert diff <= 8 * terms * (level + 1) * 2.0 ** -24


# cells a side 160 and 192: marches of 8 planes up to 295 columns' worth of 32, of 32 planes above
MF = [(5, 5, 0b111111), (3, 6, 0b111111), (3, 6, 1 | 8 | 32), (3, 6, 2 | 4 | 16)]


@pytest.mark.parametrize("n0,level,mask", MF)
def test_matrix_free_operator(oracle_mod, G, ctx, n0, level, mask):
    O, C = oracle_mod, G._capi
    rng = np.random.default_rng(mask)
    n = n0 << level
    g = G.Grid(ctx, 3, 1, level, base_level=0, n0=n0, dirichlet_mask=mask)
    k = np.exp(0.5 * rng.standard_normal(n ** 3))
    g.set_coefficient(C.FMG_K_CELL, k)
    g.assemble()
    x, b = rng.uniform(-1, 1, g.nnodes()), rng.uniform(-1, 1, (n + 1,) * 3)
    for face in range(6):  # 2 j: coordinate j (x fastest) is 0; 2 j + 1: it is n
        if mask >> face & 1:
            b[(slice(None),) * (2 - face // 2) + (n * (face % 2),)] = 0.0
    b = b.reshape(-1)
    X, B, Y = g.vector(values=x), g.vector(values=b), g.vector()
    for fp32, with_b in ((False, False), (False, True), (True, True), (2, False)):
        g.matvec_mf(X, Y, b=B if with_b else None, fp32=fp32)
        assert np.array_equal(Y.get(), O.mf_apply(n + 1, mask, k, x, b if with_b else None, fp32=fp32)), (fp32, with_b)
    # the smoothing forms, by the mixed solve's first step
    g.set_rhs(b)
    cfg = G.SolveCfg(C.FMG_METHOD_CG_MG, C.FMG_JACOBI, 0.6, 2, 2, 1, 0, 1.0, 1e-30, 0.0, 0, C.FMG_MULTIPLICATIVE)
    z = X.fill(0.0)
    g.vcycle(cfg, z, g.vector(values=b), B)
    g.matvec(z, Y)
    z = z.get()
    want = (z @ b) / (z @ Y.get()) * z
    X.fill(0.0)
    g.solve_mixed(cfg, X)
    diff = np.max(np.abs(X.get() - want)) / np.max(np.abs(want))
    print("relative difference", diff)
    assert diff <= 2 * (level + 1) * 2.0 ** -9


def test_wide_compressed_rows(oracle_mod, G, ctx):
    """A 1D chain of 400,001 unknowns, its two levels below and empty rows: the
    compressed-row kernels entry by entry (more than 150,000 rows), of the
    colours and the coarse level too, beside eight at a time below."""
    import scipy.sparse as sp
    from _hier import csr_of, oracle_of
    O, C = oracle_mod, G._capi
    rng = np.random.default_rng(2)
    sizes, mats, interp = [800], {}, {}
    for l, n in ((1, 200001), (2, 400001)):
        coarse = rng.integers(0, sizes[-1], n)
        w = rng.uniform(0.5, 1.0, n)
        w[rng.integers(0, n, n // 50)] = 0.0  # constrained: no entry in the row
        interp[l] = csr_of(sp.csr_matrix((w, (np.arange(n), coarse)), shape=(n, sizes[-1])))
        sizes.append(n)
    for l, n in enumerate(sizes):
        off = rng.uniform(-1, 0, n - 1)
        far = rng.uniform(-0.1, 0, n - 9)
        mats[l] = csr_of(sp.diags([off, off, far, far, np.full(n, 4.0)], [-1, 1, -9, 9, 0]))
    b = rng.standard_normal(sizes[-1])
    o = oracle_of(O, sizes, mats, interp, b)
    g = G.Grid.algebraic(ctx, sizes)
    for l, m in mats.items():
        g.set_matrix(l, *m)
    for l, m in interp.items():
        g.set_interpolation(l, *m, sizes[l - 1])
    g.set_rhs(b)
    for smoother, osm in ((C.FMG_JACOBI, O.JACOBI), (C.FMG_SOR, O.SOR)):
        ref = o.solve(O.solve_cfg(method=O.METHOD_MG, smoother=osm, damp=0.8, pre=1, post=2, compat=False, rtol=1e-12,
                                  maxsteps=2))
        x = g.vector()
        hist, steps, _ = g.solve(G.SolveCfg(C.FMG_METHOD_MG, smoother, 0.8, 1, 2, 1, 0, 1.0, 1e-12, 0.0, 2,
                                            C.FMG_MULTIPLICATIVE), x)
        assert steps == ref.steps and np.array_equal(hist, ref.history) and np.array_equal(x.get(), ref.x)
