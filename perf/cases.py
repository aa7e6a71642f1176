"""Performance cases of the multigrid solve path.

What a program that uses this library has it do: assemble and solve elliptic
problems on uniformly refined grids (FP64 and mixed precision, with and
without the learned damping), apply one cycle inside its own iteration, solve
many small problems at once, solve on a hierarchy it formed itself, and train
the damping network.  `listed` gives the fixed cases, `draw` further ones of
the same ranges; `prepare` builds what a program holds before the call, `run`
is one call through the public entry points, `work` what it cannot do
without, `exact` the same answer from plain torch in 64 bits.
"""
import functools
import itertools
import math
import os
import time

import numpy as np
import torch

import gnu_femlisp_b200 as G
from gnu_femlisp_b200 import _capi as C
from gnu_femlisp_b200 import adaptive
from gnu_femlisp_b200.learn import DampingNet

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(G.__file__)), "weights")
SMOOTHERS = {"jacobi": C.FMG_JACOBI, "sor": C.FMG_SOR, "ssc": C.FMG_SSC}
DAMP = {"jacobi": 0.6, "sor": 1.2, "ssc": 1.0}


def listed():
    return [
        # the smallest call: Poisson on 64 x 64 cells from one root cell, where launches and waits count
        {"name": "poisson_2d_64", "kind": "solve", "dim": 2, "order": 1, "n0": 1, "level": 6, "method": "cg",
         "smoother": "jacobi", "sweeps": 1, "field": "const"},
        # the ordinary FP64 solve: variable diffusion, assembled matrices, CG + V(1,1) Jacobi
        {"name": "diffusion_3d_fp64_128", "kind": "solve", "dim": 3, "order": 1, "n0": 1, "level": 7, "method": "cg",
         "smoother": "jacobi", "sweeps": 1, "field": "fourier"},
        # Q2 with the multicolour Gauss-Seidel/SOR smoother as the iteration, 64^3 cells
        {"name": "poisson_q2_sor_64", "kind": "solve", "dim": 3, "order": 2, "n0": 1, "level": 6, "method": "mg",
         "smoother": "sor", "sweeps": 2, "field": "const"},
        # Q2 with its default smoother, the vertex-block subspace correction, on a ragged size
        {"name": "diffusion_q2_ssc_24", "kind": "solve", "dim": 3, "order": 2, "n0": 3, "level": 3, "method": "mg",
         "smoother": "ssc", "sweeps": 1, "field": "fourier"},
        # the largest scalar solve: mixed precision and learned damping on a resident hierarchy, 256^3 cells
        {"name": "diffusion_3d_mixed_256", "kind": "mixed", "n0": 1, "level": 8, "learned": True},
        # a new coefficient field from host memory to the solution in host memory: upload, assembly, damping
        # network, judged mixed solve, download, as a time-stepping or sampling program does it
        {"name": "new_field_3d_96", "kind": "field", "n0": 3, "level": 5, "learned": True},
        # vector-Q2 elasticity, 48^3 cells (2.7 million unknowns), mixed precision with learned damping
        {"name": "elasticity_mixed_48", "kind": "elastic", "level": 4, "mixed": True, "learned": True},
        # elasticity in FP64, 12^3 cells
        {"name": "elasticity_fp64_12", "kind": "elastic", "level": 2, "mixed": False, "learned": False},
        # one cycle applied to the residual of a host's own iteration: vector up, Gauss-Seidel V(1,1), vector down
        {"name": "cycle_3d_gs_48", "kind": "cycle", "dim": 3, "order": 1, "n0": 3, "level": 4, "smoother": "sor",
         "sweeps": 1, "field": "fourier"},
        # many small problems at once: 2D fields of strong contrast with the network's damping
        {"name": "batch_2d_128x160", "kind": "batch", "level": 7, "count": 160, "learned": True},
        # a hierarchy formed by the program: a 2D mesh refined towards a corner, hanging nodes eliminated
        {"name": "adaptive_2d", "kind": "algebraic", "n0": 4, "level": 7, "smoother": "sor", "jump": 10},
        # one training step of the damping network: forward, multigrid errors, loss, gradients
        {"name": "train_step_32", "kind": "train", "n0": 1, "level": 5, "samples": 4},
    ]


def _size(rng, lo, hi, roots=(1, 2, 3, 5, 7)):
    """A root size and a level with n0 2^level spread over the logarithm of lo .. hi."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n0 = rng.choice(roots)
    return n0, max(1, int(math.log2(n / n0) + 0.5 - 1e-9)) if n0 * 2 <= hi else 1


def draw(rng):
    deviation = round(rng.uniform(0.4, 1.2), 2)  # of the logarithm of the coefficient field
    kind = rng.choice(["solve", "solve", "q2", "mixed", "field", "elastic", "cycle", "batch", "algebraic", "train"])
    if kind == "solve":
        dim = rng.choice([2, 3])
        n0, level = _size(rng, 8, 1024) if dim == 2 else _size(rng, 8, 128)
        smoother = rng.choice(["jacobi", "jacobi", "sor"])
        return {"kind": "solve", "dim": dim, "order": 1, "n0": n0, "level": level,
                "method": "cg" if smoother == "jacobi" else "mg", "smoother": smoother, "sweeps": rng.choice([1, 2]),
                "field": rng.choice(["const", "fourier"]), "deviation": deviation}
    if kind == "q2":
        n0, level = _size(rng, 6, 48, (1, 2, 3))
        smoother = rng.choice(["jacobi", "sor", "ssc"])
        return {"kind": "solve", "dim": 3, "order": 2, "n0": n0, "level": level,
                "method": "cg" if smoother == "jacobi" else "mg", "smoother": smoother, "sweeps": rng.choice([1, 2]),
                "field": rng.choice(["const", "fourier"]), "deviation": deviation}
    if kind in ("mixed", "field"):
        n0, level = _size(rng, 16, 192 if kind == "mixed" else 128)
        return {"kind": kind, "n0": n0, "level": level, "learned": rng.random() < 0.7, "deviation": deviation}
    if kind == "elastic":
        mixed = rng.random() < 0.6
        return {"kind": "elastic", "level": rng.choice([1, 2, 3]), "mixed": mixed, "learned": rng.random() < 0.5,
                "deviation": round(deviation / 2, 2)}
    if kind == "cycle":
        order = rng.choice([1, 1, 2])
        n0, level = _size(rng, 6, 96 if order == 1 else 32, (1, 2, 3, 5, 7) if order == 1 else (1, 2, 3))
        return {"kind": "cycle", "dim": 3, "order": order, "n0": n0, "level": level,
                "smoother": rng.choice(["jacobi", "sor"]), "sweeps": rng.choice([1, 2]), "field": "fourier",
                "deviation": deviation}
    if kind == "batch":
        level = rng.choice([5, 6, 7])
        return {"kind": "batch", "level": level, "count": int(2 ** rng.uniform(2, 7.2)), "learned": rng.random() < 0.5}
    if kind == "algebraic":
        return {"kind": "algebraic", "n0": rng.choice([3, 4, 5]), "level": rng.choice([3, 4, 5, 6]),
                "smoother": rng.choice(["jacobi", "sor"]), "jump": rng.choice([1, 3, 10, 30, 100])}
    n0, level = _size(rng, 8, 40, (1, 3, 5))
    return {"kind": "train", "n0": n0, "level": level, "samples": rng.choice([1, 2, 4]), "deviation": deviation}


# ------------------------------------------------------------ what a program holds
@functools.lru_cache(maxsize=None)
def _context():
    return G.Context(0)


@functools.lru_cache(maxsize=None)
def _net(name):
    return DampingNet.load(_context(), os.path.join(WEIGHTS, name))


def _base(case):
    """The coarsest level: about 4 cells a side in 3D (3 for elasticity), one root mesh in 2D."""
    dim = case.get("dim", 2 if case["kind"] == "batch" else 3)
    if case["kind"] == "elastic" or dim == 2 and case["kind"] != "batch":
        return 0
    most, b = 4, 0
    while b < case["level"] - 1 and case.get("n0", 1) << (b + 1) <= most:
        b += 1
    return b


def _cells(case):
    return (3 if case["kind"] == "elastic" else case.get("n0", 1)) << case["level"]


def _log_field(n, dim, seed, modes=64):
    """64 random Fourier modes with 1 <= |kappa| <= 10 at the cell centres, mean 0 and deviation 1 (axes z, y, x)."""
    r = np.random.default_rng(seed)
    direc = r.standard_normal((modes, dim))
    kappa = r.uniform(1, 10, modes)[:, None] * direc / np.linalg.norm(direc, axis=1, keepdims=True)
    coef = torch.as_tensor(r.standard_normal(modes) * np.exp(2j * np.pi * r.uniform(0, 1, modes)), device="cuda")
    xc = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    e = [torch.exp(2j * math.pi * torch.as_tensor(kappa[:, k], device="cuda")[:, None] * xc[None, :]) for k in range(dim)]
    left = coef[:, None]
    for k in range(dim - 1, 0, -1):
        left = (left[:, :, None] * e[k][:, None, :]).reshape(modes, -1)
    f = (left.T @ e[0]).real.reshape(-1)
    f = f - f.mean()
    return f / f.std(correction=0)


def _coefficient(case, seed):
    """The cell coefficients (x fastest), a device tensor; None for the constant 1."""
    if case["kind"] == "elastic":
        return torch.exp(case.get("deviation", 0.5) * _log_field(_cells(case), 3, seed))
    if case.get("field") == "const":
        return None
    return torch.exp(case.get("deviation", 1.0) * _log_field(_cells(case), case.get("dim", 3), seed))


def _block_fields(case, seed):
    """count fields of 8 x 8 blocks with log10 k ~ U[-3, 3]."""
    n = _cells(case)
    v = np.random.default_rng(seed).uniform(-3, 3, (case["count"], 8, 8))
    return 10.0 ** np.kron(v, np.ones((1, n // 8, n // 8))).reshape(case["count"], -1)


def _source_rhs(case, seed):
    """A nodal load h^d f with f = 1 + three sine modes, zero on the boundary (the rhs of a constant-coefficient problem)."""
    n, dim, order = _cells(case), case["dim"], case["order"]
    m = order * n + 1
    x = np.linspace(0.0, 1.0, m)
    r = np.random.default_rng(seed)
    f = np.ones((m,) * dim)
    for _ in range(3):
        t = np.array(r.standard_normal())
        for _ in range(dim):
            t = np.multiply.outer(t, np.sin(math.pi * r.integers(1, 4) * x))
        f += t
    edge = np.zeros((m,) * dim, bool)
    for k in range(dim):
        edge[(slice(None),) * k + ([0, m - 1],)] = True
    f[edge] = 0.0
    return f.reshape(-1) * (1.0 / n) ** dim


def _cfg(case, method, maxsteps=200):
    smoother = case.get("smoother", "jacobi")
    sweeps = 2 if case["kind"] == "elastic" else case.get("sweeps", 1)
    damp = 1.0 if smoother == "sor" and case["kind"] in ("cycle", "algebraic") else DAMP[smoother]
    return G.SolveCfg(method, SMOOTHERS[smoother], damp, sweeps, sweeps, 1, 0, 1.0, 1e-10, 0.0, maxsteps,
                      C.FMG_MULTIPLICATIVE)


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _grid(case, seed, coefficient=True):
    ctx = _context()
    if case["kind"] == "elastic":
        g = G.Grid(ctx, 3, 2, case["level"], 0, n0=3, ncomp=3, dirichlet_mask=0b000001)
        g.set_coefficient(C.FMG_F_VEC, [0.0, 0.0, -1.0])
        g.set_coefficient(C.FMG_LAMBDA_MU_CELL, _coefficient(case, seed).cpu().numpy())
    else:
        g = G.Grid(ctx, case.get("dim", 3), case.get("order", 1), case["level"], _base(case), n0=case.get("n0", 1))
        k = _coefficient(case, seed) if coefficient else None
        if k is not None:
            g.set_coefficient(C.FMG_K_CELL, k.cpu().numpy())
    return g


@functools.lru_cache(maxsize=8)
def _hierarchy(n0, level, jump):
    """k = jump in the quarter x, y > 1/2 and 1 elsewhere."""
    return adaptive.hierarchy(n0=n0, levels=level, kcoef=lambda x, y: 1.0 + (jump - 1.0) * (x > 0.5) * (y > 0.5))[:4]


def _algebraic_rhs(case, seed):
    rhs = _hierarchy(case["n0"], case["level"], case["jump"])[3]
    return rhs * np.random.default_rng(seed).uniform(0.5, 1.5, rhs.size)


def _with_history(s):
    """Room for the residual norms of the most steps a solve may take, zero beyond the last one."""
    s["history"] = np.zeros(s["cfg"].maxsteps + 2)
    return s


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    if kind == "algebraic":
        sizes, mats, interp, _ = _hierarchy(case["n0"], case["level"], case["jump"])
        g = G.Grid.algebraic(ctx, sizes)
        for l, m in mats.items():
            g.set_matrix(l, *m)
        for l, m in interp.items():
            g.set_interpolation(l, *m, sizes[l - 1])
        g.set_rhs(_algebraic_rhs(case, seed))
        return _with_history({"kind": kind, "grid": g, "x": g.vector(), "out": _pinned(sizes[-1]), "mixed": False,
                              "cfg": _cfg(case, C.FMG_METHOD_CG_MG)})
    if kind == "batch":
        g = G.Grid(ctx, 2, 1, case["level"], _base(case))
        batch = G.Grid.batch(g, case["count"])
        for i, k in enumerate(_block_fields(case, seed)):
            g.set_coefficient(C.FMG_K_CELL, k)
            g.assemble()
            if case["learned"]:
                _net("damping2d.fmgnet").apply(g)
            batch.batch_load(i, g)
        return {"kind": kind, "grid": batch, "x": batch.vector(), "out": _pinned(g.nnodes() * case["count"]),
                "cfg": _cfg(case, C.FMG_METHOD_CG_MG)}
    if kind == "train":
        g = _grid(case, seed).assemble()
        return {"kind": kind, "grid": g, "net": DampingNet(ctx, 3, seed=seed), "samples": case["samples"],
                "seed": seed, "cfg": _cfg(case, C.FMG_METHOD_CG_MG)}
    if kind == "field":
        g = _grid(case, seed, coefficient=False)
        k = _pinned(_cells(case) ** 3)
        k[:] = _coefficient(case, seed).cpu().numpy()
        return {"kind": kind, "grid": g, "k": k, "net": _net("damping3d.fmgnet") if case["learned"] else None,
                "x": G.Vector(g, g.top), "out": _pinned(g.nnodes()), "cfg": _cfg(case, C.FMG_METHOD_CG_MG)}
    g = _grid(case, seed).assemble()
    if kind == "solve" and case["field"] == "const":
        g.set_rhs(_source_rhs(case, seed))
    if case.get("learned"):
        _net("damping3d_elastic.fmgnet" if kind == "elastic" else "damping3d.fmgnet").apply(g)
    s = {"kind": kind, "grid": g, "x": g.vector(), "out": _pinned(g.nnodes() * g.nc),
         "mixed": kind == "mixed" or bool(case.get("mixed")), "judge": int(kind == "mixed" and case["learned"]),
         "cfg": _cfg(case, C.FMG_METHOD_MG if case.get("method") == "mg" else C.FMG_METHOD_CG_MG)}
    if kind == "cycle":
        s.update(b=g.vector(), r=g.vector(), residual=_pinned(g.nnodes()))
        s["residual"][:] = _source_rhs(case, seed)
    return _with_history(s)


# ------------------------------------------------------------ one call
def run(s):
    kind, g = s["kind"], s["grid"]
    if kind == "train":
        s["net"].zero_grads()
        loss = s["net"].step(g, s["cfg"], s["samples"], s["seed"], 4)
        return {"loss": loss, "grads": s["net"].grads}
    x = s["x"]
    if kind == "cycle":  # r and b hold the residual, x the correction
        s["b"].set(s["residual"])
        s["b"].copy_to(s["r"])
        x.fill(0.0)
        g.vcycle(s["cfg"], x, s["b"], s["r"])
        return {"x": x.get(s["out"])}
    if kind == "batch":
        x.fill(0.0)
        history, steps, status = g.batch_solve(s["cfg"], x)
        return {"x": x.get(s["out"]), "history": history, "steps": steps, "status": status}
    if kind == "field":
        g.set_coefficient(C.FMG_K_CELL, s["k"])
        g.assemble()
        if s["net"] is not None:
            s["net"].apply(g)
        x.fill(0.0)
        _, _, steps, status = g.solve_mixed(s["cfg"], x, judge=int(s["net"] is not None))
        return {"x": x.get(s["out"]), "steps": steps, "status": status}
    x.fill(0.0)
    if s["mixed"]:
        _, _, steps, status = g.solve_mixed(s["cfg"], x, judge=s["judge"])
        return {"x": x.get(s["out"]), "steps": steps, "status": status}
    history, steps, status = g.solve(s["cfg"], x)
    s["history"][:history.size] = history
    return {"x": x.get(s["out"]), "history": s["history"], "steps": steps, "status": status}


# ------------------------------------------------------------ what a call cannot do without
def work(case):
    """Every step streams the level matrices once per application (operator, residual and smoothing sweeps; the
    cell coefficients in their place where the operator is matrix-free) and about 20 vector passes; the steps are
    those such problems take.  Levels below the top add 1/7 (1/3 in 2D)."""
    kind, n = case["kind"], _cells(case) if case["kind"] != "algebraic" else 0
    if kind == "algebraic":
        sizes, mats, _, _ = _hierarchy(case["n0"], case["level"], case["jump"])
        nnz = sum(len(m[1]) for m in mats.values())
        per = 4 * 12 * nnz + 20 * 8 * sum(sizes)
        return {"bytes": 9 * per, "flops": 9 * 8 * nnz}
    dim, order = case.get("dim", 2 if kind == "batch" else 3), 2 if kind == "elastic" else case.get("order", 1)
    nodes = (order * n + 1) ** dim
    nnz = nodes * ((3.0 if order == 1 else 4.0) ** dim)  # Q2 rows have 3 or 5 entries a direction
    levels = 2.0 ** dim / (2.0 ** dim - 1)
    sweeps = 2 if kind == "elastic" else case.get("sweeps", 1)
    if kind == "train":
        convolutions = 3 * 2 * 27 * (16 * 32 + 32 * 32 + 32) * nodes * levels
        cycles = case["samples"] * (4 + 3)
        return {"bytes": cycles * 3 * 8 * nnz * levels + 3 * 2 * 80 * nodes * levels,
                "flops": convolutions + cycles * 6 * nnz * levels}
    if kind in ("mixed", "field"):
        steps = 14 if case["learned"] else 18
        per = nodes * (24 + 20 + 36 + 60) + nnz / 8 * levels * 4 * 2
        w = {"bytes": steps * per, "flops": steps * 4 * 2 * nnz}
        if kind == "field":
            w["bytes"] += n ** 3 * 16 + nnz / 8 * levels * 8 + nodes * 8
            if case["learned"]:
                w["bytes"] += 2 * (32 + 64 + 64) * nodes * levels
                w["flops"] += 2 * 27 * (16 * 32 + 32 * 32 + 32) * nodes * levels
        return w
    if kind == "elastic":
        per = 9 * nnz * 8 + 9 * nnz * (4 if case["mixed"] else 8) * 2 * sweeps * levels + 20 * 24 * nodes
        return {"bytes": 18 * per, "flops": 18 * 2 * 9 * nnz * (1 + 2 * sweeps * levels)}
    if kind == "cycle":
        per = nnz * 8 * (2 * sweeps + 1) * levels + 10 * 8 * nodes
        return {"bytes": per, "flops": 2 * nnz * (2 * sweeps + 1) * levels}
    count = case.get("count", 1)
    steps = 24 if kind == "batch" else 12 if case.get("method") == "cg" else 9
    per = nnz * 8 * (1 + 2 * sweeps * levels) + 20 * 8 * nodes
    return {"bytes": count * steps * per, "flops": count * steps * 2 * nnz * (1 + 2 * sweeps * levels)}


# ------------------------------------------------------------ the answer in 64 bits
def _element(dim, order, elastic):
    """The reference element's stiffness (unit cell, unit coefficient; lambda = mu = 1 where elastic) and load."""
    t, w = np.polynomial.legendre.leggauss(order + 1)
    pts, wts = (t + 1) / 2, w / 2
    nodes = np.linspace(0.0, 1.0, order + 1)
    val, der = np.empty((order + 1, order + 1)), np.empty((order + 1, order + 1))
    for a in range(order + 1):
        p = np.poly1d(np.poly(np.delete(nodes, a)) / np.prod(nodes[a] - np.delete(nodes, a)))
        val[a], der[a] = p(pts), p.deriv()(pts)
    local = [t[::-1] for t in itertools.product(range(order + 1), repeat=dim)]  # x fastest
    nl = len(local)
    K, F = np.zeros((nl, nl, dim, dim)), np.zeros(nl)
    for q in itertools.product(range(order + 1), repeat=dim):
        wq = np.prod([wts[i] for i in q])
        phi = np.array([np.prod([val[a[k], q[k]] for k in range(dim)]) for a in local])
        grad = np.array([[np.prod([(der if j == k else val)[a[j], q[j]] for j in range(dim)]) for k in range(dim)]
                         for a in local])
        K += wq * np.einsum("ak,bl->abkl", grad, grad)
        F += wq * phi
    if not elastic:
        return np.einsum("abkk->ab", K), F, local
    E = K + np.swapaxes(K, 2, 3) + np.einsum("abjj,kl->abkl", K, np.eye(dim))
    return E.transpose(0, 2, 1, 3).reshape(nl * dim, nl * dim), F, local


def _pcg(apply, diag, b, limit_s=16.0, rtol=1e-14):
    """Jacobi-preconditioned CG on [problems, unknowns]; None when it takes too long."""
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz = z.clone(), (r * z).sum(1, keepdim=True)
    stop, began = rtol * b.norm(dim=1), time.monotonic()
    for it in range(100000):
        a = apply(p)
        pa = (p * a).sum(1, keepdim=True)
        al = torch.where(pa > 0, rz / pa, torch.zeros_like(pa))
        x += al * p
        r -= al * a
        z = r / diag
        new = (r * z).sum(1, keepdim=True)
        p = z + torch.where(rz > 0, new / rz, torch.zeros_like(rz)) * p
        rz = new
        if it % 25 == 24:
            if bool((r.norm(dim=1) <= stop).all()):
                return x
            if time.monotonic() - began > limit_s:
                return None
    return None


def _exact_structured(case, seed):
    kind, n = case["kind"], _cells(case)
    elastic = kind == "elastic"
    dim, order = case.get("dim", 2 if kind == "batch" else 3), 2 if elastic else case.get("order", 1)
    nc, m, h, count = 3 if elastic else 1, order * n + 1, 1.0 / n, case.get("count", 1)
    if elastic and n > 24 or m ** dim > 3e6 and order == 2 or m ** dim > 2e7:
        return None
    K, F, local = _element(dim, order, elastic)
    K = torch.as_tensor(K, device="cuda") * h ** (dim - 2)
    if kind == "batch":
        k = torch.as_tensor(_block_fields(case, seed), device="cuda")
    else:
        k = _coefficient(case, seed)
        k = torch.ones(1, n ** dim, device="cuda", dtype=torch.float64) if k is None else k.reshape(1, -1)
    shape = (count,) + (m,) * dim + (nc,)
    cuts = [tuple([slice(None)] + [slice(a[dim - 1 - j], a[dim - 1 - j] + order * (n - 1) + 1, order)
                                   for j in range(dim)]) for a in local]

    def scatter(per_cell, into):
        for a, cut in enumerate(cuts):
            into[cut] += per_cell[..., a * nc:(a + 1) * nc].reshape((count,) + (n,) * dim + (nc,))
        return into

    free = torch.ones(shape, device="cuda", dtype=torch.float64)
    if elastic:
        free[:, :, :, 0] = 0.0  # the face x = 0
    else:
        for j in range(1, dim + 1):
            free.index_fill_(j, torch.tensor([0, m - 1], device="cuda"), 0.0)

    def apply(v):
        v = v.reshape(shape)
        cells = torch.cat([v[cut].reshape(count, -1, nc) for cut in cuts], dim=2)
        y = scatter((cells @ K) * k[..., None], torch.zeros(shape, device="cuda", dtype=torch.float64))
        return (y * free).reshape(count, -1)

    diag = scatter(k[..., None] * torch.diagonal(K), torch.zeros_like(free))
    diag = torch.where(free > 0, diag, torch.ones_like(diag)).reshape(count, -1)
    if kind == "solve" and case["field"] == "const":
        b = torch.as_tensor(_source_rhs(case, seed), device="cuda").reshape(1, -1)
    else:
        load = np.zeros((len(local), nc))
        load[:, nc - 1] = F * h ** dim * (-1.0 if elastic else 1.0)
        load = torch.as_tensor(load.reshape(-1), device="cuda").expand(count, n ** dim, -1)
        b = (scatter(load, torch.zeros_like(free)) * free).reshape(count, -1)
    x = _pcg(apply, diag, b)
    return None if x is None else x.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "cycle"):  # the network's BF16 values, one cycle's own iterate: no value in 64 bits
        return None
    if kind == "algebraic":
        start, index, value = _hierarchy(case["n0"], case["level"], case["jump"])[1][case["level"]]
        A = torch.sparse_csr_tensor(torch.as_tensor(start), torch.as_tensor(index.astype(np.int64)),
                                    torch.as_tensor(value)).to("cuda")
        b = torch.as_tensor(_algebraic_rhs(case, seed), device="cuda").reshape(1, -1)
        rows = torch.repeat_interleave(torch.arange(len(start) - 1), torch.as_tensor(np.diff(start)))
        on = torch.as_tensor(index.astype(np.int64)) == rows
        diag = torch.as_tensor(value)[on].to("cuda").reshape(1, -1)
        x = _pcg(lambda v: (A @ v.reshape(-1, 1)).reshape(1, -1), diag, b)
        x = None if x is None else x.reshape(-1)
    else:
        x = _exact_structured(case, seed)
    if x is None:
        return None
    none = {"x": x, "steps": None, "status": None}
    return none if kind in ("mixed", "field") or case.get("mixed") else {**none, "history": None}
