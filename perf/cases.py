"""Performance cases: the calls that programs on this framework make, over the
range of sizes they make them at.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call, ``run(state)``
is one pass through the public entry points, ``work(case)`` the bytes and
floating-point operations that pass cannot do without, and ``exact(case, seed)``
its result in 64 bits from plain NumPy and PyTorch.

Kinds of case:

poisson    right-hand side, fast-diagonalisation solve and backward transform
           of a Dirichlet Poisson or Helmholtz problem (all FP64)
roundtrip  backward then forward transform of a batch of fields: FP64 data (the
           default precision), FP32 data with split-BF16 operators, or FP64
           data of a space with inhomogeneous Dirichlet values
helmholtz  a batch of Helmholtz solves of uneven sizes in one call
operator   the matrix-free variable-coefficient operator applied to a batch
pcg        batched FP64 PCG on that operator
mixed      the mixed-precision solver on that operator, from zero or from the
           learned initial guess
train      one training step of the spectral neural operator
"""

from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

import jaxfun_gb300
from jaxfun_gb300.galerkin import DIRICHLET, Chebyshev, FunctionSpace, Legendre, TensorProduct
from jaxfun_gb300.la import MixedVarCoefSolver, VarCoefMatrix, pcg, poisson_tpmatrices
from jaxfun_gb300.la.helmholtz import UnevenHelmholtzSolver
from jaxfun_gb300.sno import train as sno_train
from jaxfun_gb300.sno.model import CIN, COUT, SNO, SNOConfig

F64 = torch.float64
FAMILIES = {"legendre": Legendre, "chebyshev": Chebyshev}
#: Dirichlet values of the lifted round trips at x = -1 and x = 1 (functions of y)
LIFT_LEFT, LIFT_RIGHT = 1.0, 2.0
#: iterations of the inner PCG that a solve of these tolerances takes, for work()
ITERATIONS = {2: 90, 3: 180}
HELMHOLTZ_SIZES = tuple(range(32, 513, 16))


def listed():
    return [
        # the smallest call: one small problem, three calls, bound by latency
        {"name": "poisson2d_one", "kind": "poisson", "family": "legendre", "ndim": 2, "N": 64,
         "batch": 1, "alpha2": 0.0},
        # many small problems of one size (a parameter study)
        {"name": "poisson2d_many", "kind": "poisson", "family": "legendre", "ndim": 2, "N": 64,
         "batch": 1024, "alpha2": 0.0},
        # a few 3-D Helmholtz problems of an odd size (an implicit time step)
        {"name": "helmholtz3d_odd", "kind": "poisson", "family": "chebyshev", "ndim": 3, "N": 51,
         "batch": 4, "alpha2": 37.0},
        # FP64 transforms there and back (the default precision), as in a
        # pseudo-spectral step
        {"name": "roundtrip3d_f64", "kind": "roundtrip", "family": "chebyshev", "ndim": 3,
         "N": 128, "batch": 8, "precision": "f64"},
        # the same at the largest size, FP32 data on split-BF16 operators
        {"name": "roundtrip3d_bf16x3", "kind": "roundtrip", "family": "chebyshev", "ndim": 3,
         "N": 256, "batch": 16, "precision": "bf16x3"},
        # fields with inhomogeneous Dirichlet values, ragged size
        {"name": "roundtrip2d_lifted", "kind": "roundtrip", "family": "legendre", "ndim": 2,
         "N": 150, "batch": 24, "precision": "lifted"},
        # 1024 problems of 31 sizes between 32 and 512 in one call
        {"name": "helmholtz_uneven", "kind": "helmholtz", "family": "chebyshev", "count": 1024,
         "top": 512, "plan": 0},
        # the variable-coefficient operator on a batch, as in an outer iteration
        {"name": "operator2d", "kind": "operator", "ndim": 2, "N": 256, "batch": 32},
        # plain FP64 PCG on a few problems
        {"name": "pcg2d_f64", "kind": "pcg", "ndim": 2, "N": 128, "batch": 8, "tol": 5e-12},
        # the headline workload: 128 problems, learned guess, mixed precision
        {"name": "mixed2d_learned", "kind": "mixed", "ndim": 2, "N": 256, "batch": 128,
         "guess": True, "tol": 1e-11},
        # 3-D problems from a zero start
        {"name": "mixed3d", "kind": "mixed", "ndim": 3, "N": 128, "batch": 8, "guess": False,
         "tol": 1e-12},
        # one training step of the network behind the learned guess
        {"name": "sno_train", "kind": "train", "n": 64, "width": 64, "modes": 32, "batch": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "roundtrip", "roundtrip", "helmholtz", "operator",
                       "operator", "pcg", "mixed", "mixed", "train"])
    if kind == "poisson":
        nd = rng.choice([2, 2, 3])
        N = rng.randint(17, 200) if nd == 2 else rng.randint(13, 80)
        return {"kind": kind, "family": rng.choice(["legendre", "chebyshev"]), "ndim": nd, "N": N,
                "batch": min(_log_int(rng, 1, 1024), max(1, 4_000_000 // N**nd)),
                "alpha2": rng.choice([0.0, round(rng.uniform(0.5, 400.0), 2)])}
    if kind == "roundtrip":
        precision = rng.choice(["f64", "bf16x3", "lifted"])
        family = rng.choice(["legendre", "chebyshev"])
        if precision == "lifted":
            N = rng.randint(20, 256)
            return {"kind": kind, "family": family, "ndim": 2, "N": N,
                    "batch": _log_int(rng, 1, max(2, 4_000_000 // N**2)), "precision": precision}
        nd = rng.choice([2, 3])
        N = rng.randint(32, 256) if nd == 2 else rng.randint(24, 160)
        if precision == "bf16x3":
            N = max(32, N // 8 * 8)  # rows of 16 bytes, as that precision asks for
        return {"kind": kind, "family": family, "ndim": nd, "N": N,
                "batch": _log_int(rng, 1, max(2, min(1024, 16_000_000 // N**nd))),
                "precision": precision}
    if kind == "helmholtz":
        return {"kind": kind, "family": rng.choice(["legendre", "chebyshev"]),
                "count": _log_int(rng, 16, 512), "top": rng.choice([128, 256, 384]),
                "plan": rng.randint(1, 999)}
    if kind == "operator":
        nd = rng.choice([2, 3])
        N = rng.randint(24, 256) if nd == 2 else rng.randint(12, 96)
        return {"kind": kind, "ndim": nd, "N": N,
                "batch": _log_int(rng, 1, max(2, min(256, 2_000_000 // N**nd)))}
    if kind == "pcg":
        nd = rng.choice([2, 2, 3])
        N = rng.randint(24, 160) if nd == 2 else rng.randint(12, 40)
        return {"kind": kind, "ndim": nd, "N": N,
                "batch": _log_int(rng, 1, max(2, min(64, 400_000 // N**nd))), "tol": 5e-12}
    if kind == "mixed":
        nd = rng.choice([2, 2, 3])
        N = 4 * (rng.randint(12, 64) if nd == 2 else rng.randint(6, 24))
        return {"kind": kind, "ndim": nd, "N": N,
                "batch": _log_int(rng, 1, max(2, min(128, 4_000_000 // N**nd))),
                "guess": False, "tol": 1e-11 if nd == 2 else 1e-12}
    return {"kind": kind, "n": 32, "width": rng.choice([32, 64]), "modes": rng.choice([16, 24]),
            "batch": rng.randint(4, 32)}


# ---------------------------------------------------------------------------
# what a program keeps
# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=1)
def _solver_stream():
    """The stream the solvers run on: one that can be captured."""
    return torch.cuda.Stream()


@functools.lru_cache(maxsize=16)
def _space(family, ndim, N, precision=""):
    if precision == "lifted":
        D = FunctionSpace(N, FAMILIES[family], bcs=DIRICHLET)
        X = FunctionSpace(N, FAMILIES[family],
                          bcs={"left": {"D": LIFT_LEFT}, "right": {"D": LIFT_RIGHT}})
        return TensorProduct(X, D)
    if precision:
        return TensorProduct(*([FAMILIES[family](N)] * ndim))
    return TensorProduct(*([FunctionSpace(N, FAMILIES[family], bcs=DIRICHLET)] * ndim))


@functools.lru_cache(maxsize=16)
def _poisson_matrix(family, ndim, N, alpha2):
    A = poisson_tpmatrices(_space(family, ndim, N), alpha2)
    A.lu_factor()
    return A


@functools.lru_cache(maxsize=4)
def _helmholtz_solver(family, count, top, plan):
    Ns, alphas = _helmholtz_plan(count, top, plan)
    return UnevenHelmholtzSolver(family, Ns, alphas)


def _helmholtz_plan(count, top, plan):
    rng = np.random.default_rng(plan)
    sizes = [N for N in HELMHOLTZ_SIZES if N <= top]
    return rng.choice(sizes, size=count), rng.uniform(0.0, 50.0, size=count)


@functools.lru_cache(maxsize=2)
def _network(batch):
    weights = os.path.join(os.path.dirname(jaxfun_gb300.__file__), "sno", "weights",
                           "sno_varcoef2d_N256.npz")
    return sno_train.load(weights, batch=batch), sno_train.GridMaps()


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(gen, shape, dtype=F64):
    return torch.randn(shape, generator=gen, dtype=dtype, device="cuda")


def _decay(N, power, ndim):
    """(1 + k)^-power per axis, as the coefficients of smooth fields fall off."""
    v = (1.0 + torch.arange(N, dtype=F64, device="cuda")) ** -power
    out = v
    for _ in range(ndim - 1):
        out = out[..., None] * v
    return out


def _field_values(family, N, coef, ndim):
    return _kron([_dev(_vander(family, N, N))] * ndim, coef)


def _coefficient(seed, ndim, N, batch):
    """kappa = exp(g), g a Gaussian random field standardised per problem, and
    the forcing f, both on the Legendre-Gauss grid."""
    gen = _generator(seed)
    k2 = torch.arange(N, dtype=F64, device="cuda") ** 2
    s = k2
    for _ in range(ndim - 1):
        s = s[..., None] + k2
    axes = tuple(range(1, ndim + 1))
    g = _field_values("legendre", N, _randn(gen, (batch,) + (N,) * ndim) * (1.0 + s) ** -1.5, ndim)
    g = (g - g.mean(dim=axes, keepdim=True)) / g.std(dim=axes, keepdim=True)
    f = _field_values("legendre", N, _randn(gen, (batch,) + (N,) * ndim) * _decay(N, 2.0, ndim),
                      ndim)
    return g, f


def _varcoef_inputs(case, seed):
    nd, N, B = case["ndim"], case["N"], case["batch"]
    g, f = _coefficient(seed, nd, N, B)
    b = _kron([_dev(_scalar_product("legendre", N))] * nd, f)
    return g, f, b


def _helmholtz_rhs(case, seed):
    """Packed right-hand sides, in the solver's order: by size, then by problem."""
    Ns, _ = _helmholtz_plan(case["count"], case["top"], case["plan"])
    gen = _generator(seed)
    out = []
    for N in sorted(set(Ns.tolist())):
        cnt = int((Ns == N).sum())
        Q = _dev(_scalar_product(case["family"], N) @ _vander(case["family"], N, N))
        c = _randn(gen, (cnt, N, N)) * _decay(N, 2.0, 2)
        out.append((Q @ c @ Q.T).reshape(-1))
    return torch.cat(out)


def _roundtrip_input(case, seed):
    N, nd, B = case["N"], case["ndim"], case["batch"]
    gen = _generator(seed)
    if case["precision"] == "bf16x3":
        c = _randn(gen, (B,) + (N,) * nd, torch.float32)
        return c.mul_(_decay(N, 1.0, nd).float())
    n = N - 2 if case["precision"] == "lifted" else N
    return _randn(gen, (B,) + (n,) * nd) * _decay(n, 1.0, nd)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        fam, nd, N = case["family"], case["ndim"], case["N"]
        c = _randn(_generator(seed), (case["batch"],) + (N,) * nd) * _decay(N, 2.0, nd)
        f = _field_values(fam, N, c, nd)
        return {"kind": kind, "T": _space(fam, nd, N), "f": f[0] if case["batch"] == 1 else f,
                "A": _poisson_matrix(fam, nd, N, case["alpha2"])}
    if kind == "roundtrip":
        lifted = case["precision"] == "lifted"
        return {"kind": kind, "c": _roundtrip_input(case, seed),
                "T": _space(case["family"], case["ndim"], case["N"], case["precision"]),
                "precision": "f64" if lifted else case["precision"]}
    if kind == "train":
        with torch.cuda.stream(_solver_stream()):
            model, x, target = _train_inputs(case, seed)
        return {"kind": kind, "model": model, "x": x, "target": target}
    with torch.cuda.stream(_solver_stream()):
        if kind == "helmholtz":
            solver = _helmholtz_solver(case["family"], case["count"], case["top"], case["plan"])
            return {"kind": kind, "solver": solver, "b": _helmholtz_rhs(case, seed)}
        g, f, b = _varcoef_inputs(case, seed)
        T = _space("legendre", case["ndim"], case["N"])
        A = VarCoefMatrix(T, torch.exp(g))
        state = {"kind": kind, "A": A, "b": b}
        if kind == "operator":
            n = case["N"] - 2
            state["u"] = b.new_empty(b.shape).copy_(
                _randn(_generator(seed + 1), b.shape) * _decay(n, 1.0, case["ndim"]))
        elif kind == "pcg":
            state.update(tol=case["tol"], M=_poisson_matrix("legendre", case["ndim"], case["N"],
                                                            0.0).lu_factor())
        else:
            M = _poisson_matrix("legendre", case["ndim"], case["N"], 0.0).lu_factor()
            state.update(tol=case["tol"], solver=MixedVarCoefSolver(A, M), network=None)
            if case["guess"]:
                state.update(network=_network(case["batch"]), g=g, f=f)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "poisson":
        T = state["T"]
        c = state["A"].solve(T.scalar_product(state["f"]))
        return c, T.backward(c)
    if kind == "roundtrip":
        u = state["T"].backward(state["c"], precision=state["precision"])
        return u, state["T"].forward(u, precision=state["precision"])
    with torch.cuda.stream(_solver_stream()):
        if kind == "helmholtz":
            return state["solver"].solve_packed(state["b"], tol=1e-11)[0]
        if kind == "operator":
            return state["A"] @ state["u"]
        if kind == "pcg":
            return pcg(state["A"], state["b"], M=state["M"], tol=state["tol"])[0]
        if kind == "mixed":
            guess = None
            if state["network"] is not None:
                model, maps = state["network"]
                X, s = sno_train.features(state["g"], state["f"], maps)
                guess = sno_train.initial_guess(model, maps, X, s)
            return state["solver"].solve(state["b"], tol=state["tol"], guess=guess)[0]
        model = state["model"]
        Bt = model.set_input(state["x"])
        model.forward(Bt)
        loss = model.backward(Bt, state["target"])
        model.adam(1e-3)
        return {"loss": loss, "grads": model.grads, "params": model.params}


def _train_inputs(case, seed):
    cfg = SNOConfig(n=case["n"], width=case["width"], modes=case["modes"], batch=case["batch"])
    model = SNO(cfg, seed=0)
    gen = _generator(seed)
    n, B = case["n"], case["batch"]
    low = min(n, 12)
    coef = torch.zeros((2 * B, n, n), dtype=F64, device="cuda")
    coef[:, :low, :low] = _randn(gen, (2 * B, low, low)) * _decay(low, 1.5, 2)
    v = _field_values("legendre", n, coef, 2)
    v = v / v.std(dim=(1, 2), keepdim=True)
    x = torch.zeros((B, n, n, CIN), dtype=F64, device="cuda")
    node = _dev(_nodes("legendre", n)[0])
    x[..., 0], x[..., 1] = v[:B], v[B:]
    x[..., 2], x[..., 3] = node[:, None], node[None, :]
    target = 0.1 * v[B:] * torch.exp(-0.5 * v[:B])
    return (model, x.reshape(B * n * n, CIN).to(torch.bfloat16),
            target.float().reshape(-1).contiguous())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _apply_flops(ndim, rows, cols, batch):
    """Separable apply, last axis first: 2 M P K per pass."""
    shape, total = [cols] * ndim, 0.0
    for t in range(ndim):
        shape[ndim - 1 - t] = rows
        total += 2.0 * cols * math.prod(shape)
    return total * batch


def _operator_flops(ndim, N, batch):
    """Gradient to the grid, coefficient, and back: per component one separable
    apply each way, shared passes counted once."""
    n, q = N - 2, N
    if ndim == 2:
        passes = 4.0 * q * n * n + 4.0 * q * q * n
    else:
        passes = 4.0 * q * n**3 + 6.0 * q * q * n * n + 6.0 * q**3 * n
    return batch * (2 * passes + ndim * q**ndim)


def work(case):
    kind = case["kind"]
    if kind == "train":
        P, NM, C, B = case["n"] ** 2, case["modes"] ** 2, case["width"], case["batch"]
        layer = 2.0 * B * C * (2 * NM * P + NM * C + P * C)
        forward = 4 * layer + 2.0 * B * P * C * (CIN + C + COUT)
        params = 4 * (NM * C * C + C * C + C) + C * CIN + C * C + COUT * C
        return {"bytes": 2.0 * B * P * CIN + 4.0 * B * P + 28.0 * params, "flops": 3 * forward}
    if kind == "helmholtz":
        Ns, _ = _helmholtz_plan(case["count"], case["top"], case["plan"])
        n = Ns.astype(np.float64) - 2
        return {"bytes": 16.0 * float((n**2).sum()), "flops": 8.0 * float((n**3).sum())}
    nd, N, B = case["ndim"], case["N"], case["batch"]
    n = N - 2
    if kind == "poisson":
        flops = (_apply_flops(nd, n, N, B) + 2 * _apply_flops(nd, n, n, B)
                 + _apply_flops(nd, N, n, B))
        return {"bytes": 8.0 * B * (2 * N**nd + n**nd), "flops": flops}
    if kind == "roundtrip":
        m = n if case["precision"] == "lifted" else N
        size = 4 if case["precision"] == "bf16x3" else 8
        return {"bytes": float(size) * B * (2 * m**nd + N**nd),
                "flops": _apply_flops(nd, N, m, B) + _apply_flops(nd, m, N, B)}
    apply = _operator_flops(nd, N, B)
    if kind == "operator":
        return {"bytes": 8.0 * B * (2 * n**nd + N**nd), "flops": apply}
    iteration = apply + 2 * _apply_flops(nd, n, n, B)
    return {"bytes": 8.0 * B * (2 * n**nd + N**nd), "flops": ITERATIONS[nd] * iteration}


# ---------------------------------------------------------------------------
# the results in 64 bits, from NumPy and PyTorch alone
# ---------------------------------------------------------------------------


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device="cuda")


def _kron(mats, x):
    """(x_ax mats[ax]) x over the trailing axes."""
    nd = len(mats)
    for t, m in enumerate(reversed(mats)):
        ax = x.ndim - 1 - t
        x = (x.movedim(ax, -1) @ m.T).movedim(-1, ax)
    return x.contiguous() if nd else x


@functools.lru_cache(maxsize=64)
def _legendre_rule(N):
    """Gauss-Legendre nodes, weights, and the first N polynomials and their
    derivatives at the nodes, by recurrences in extended precision."""
    k = np.arange(1, N + 1, dtype=np.longdouble)
    x = -np.cos(np.pi * (4 * k - 1) / (4 * N + 2))
    for step in range(5):
        V = np.polynomial.legendre.legvander(x, N)
        slope = N * (x * V[:, N] - V[:, N - 1]) / (x * x - 1)
        if step < 4:
            x = x - V[:, N] / slope
    D = np.zeros_like(V)
    for j in range(1, N + 1):
        D[:, j] = (2 * j - 1) * V[:, j - 1] + (D[:, j - 2] if j > 1 else 0)
    return tuple(a.astype(np.float64) for a in (x, 2 / ((1 - x * x) * slope * slope),
                                                V[:, :N], D[:, :N]))


@functools.lru_cache(maxsize=64)
def _nodes(family, N):
    if family == "legendre":
        return _legendre_rule(N)[:2]
    k = np.arange(N)
    return -np.cos((2 * k + 1) * np.pi / (2 * N)), np.full(N, np.pi / N)


@functools.lru_cache(maxsize=64)
def _vander(family, Nq, N):
    """Values of the first N <= Nq polynomials at the Nq Gauss nodes."""
    if family == "legendre":
        return _legendre_rule(Nq)[2][:, :N]
    m = (np.arange(N)[None, :] * (2 * Nq - 2 * np.arange(Nq)[:, None] - 1)) % (4 * Nq)
    return np.cos(m * (np.pi / (2 * Nq)))


def _dirichlet(V):
    return V[:, :-2] - V[:, 2:]


@functools.lru_cache(maxsize=64)
def _scalar_product(family, N):
    """(dim x Nq) scalar products with the Dirichlet basis."""
    return (_dirichlet(_vander(family, N, N)) * _nodes(family, N)[1][:, None]).T.copy()


@functools.lru_cache(maxsize=64)
def _galerkin(family, N):
    """Mass matrix and stiffness -(phi_j'', phi_i)_w of the Dirichlet basis."""
    S = np.eye(N - 2, N) - np.eye(N - 2, N, 2)
    i, j = np.arange(N)[:, None], np.arange(N)[None, :]
    mask = (j - i >= 2) & ((j - i) % 2 == 0)
    if family == "legendre":
        h = 2.0 / (2.0 * np.arange(N) + 1.0)
        D2 = np.where(mask, j * (j + 1.0) - i * (i + 1.0), 0.0)
    else:
        h = np.full(N, np.pi / 2)
        h[0] = np.pi
        D2 = np.where(mask, j * (j * j - i * i) * (np.pi / 2), 0.0)
    return S @ np.diag(h) @ S.T, -(S @ D2 @ S.T)


@functools.lru_cache(maxsize=64)
def _diagonalised(family, N):
    """lam, W, E with K W = M W diag(lam) and E = (M W)^-1."""
    M, K = _galerkin(family, N)
    if family == "legendre":
        Li = np.linalg.inv(np.linalg.cholesky(M))
        lam, Q = np.linalg.eigh(Li @ K @ Li.T)
        W = Li.T @ Q
        return lam, W, W.T.copy()
    lam, W = np.linalg.eig(np.linalg.solve(M, K))
    lam, W = lam.real, W.real
    return lam, W, np.linalg.inv(M @ W)


def _helmholtz_solve(family, N, ndim, alpha2, b, refine=2):
    """alpha2 (x M) u + sum of stiffness terms = b by diagonalisation, refined
    with the dense residual.  alpha2: a number, or one per leading index."""
    lam, W, E = (_dev(a) for a in _diagonalised(family, N))
    M, K = (_dev(a) for a in _galerkin(family, N))
    a2 = torch.as_tensor(alpha2, dtype=F64, device="cuda").reshape((-1,) + (1,) * ndim)
    if b.ndim == ndim:
        a2 = a2.reshape(())
    s = lam
    for _ in range(ndim - 1):
        s = s[..., None] + lam

    def residual(u):
        r = b - a2 * _kron([M] * ndim, u)
        for ax in range(ndim):
            r = r - _kron([K if i == ax else M for i in range(ndim)], u)
        return r

    u = _kron([W] * ndim, _kron([E] * ndim, b) / (a2 + s))
    for _ in range(refine):
        u = u + _kron([W] * ndim, _kron([E] * ndim, residual(u)) / (a2 + s))
    return u


def _varcoef(case, seed):
    """(matvec, right-hand side) of the case's variable-coefficient problem."""
    nd, N = case["ndim"], case["N"]
    g, _, b = _varcoef_inputs(case, seed)
    kw = torch.exp(g)
    w = _dev(_nodes("legendre", N)[1])
    for ax in range(nd):
        kw = kw * w.reshape((-1,) + (1,) * (nd - 1 - ax))
    B = _dev(_dirichlet(_vander("legendre", N, N)))
    D = _dev(_dirichlet(_legendre_rule(N)[3]))

    def matvec(u):
        out = 0.0
        for ax in range(nd):
            ops = [D if i == ax else B for i in range(nd)]
            out = out + _kron([o.T for o in ops], kw * _kron(ops, u))
        return out

    return matvec, b


def _varcoef_solve(case, seed):
    """Preconditioned conjugate gradients until the residual no longer falls."""
    nd, N = case["ndim"], case["N"]
    matvec, b = _varcoef(case, seed)
    lam, W, _ = (_dev(a) for a in _diagonalised("legendre", N))
    s = lam
    for _ in range(nd - 1):
        s = s[..., None] + lam
    axes = tuple(range(1, nd + 1))

    def precondition(r):
        return _kron([W] * nd, _kron([W.T] * nd, r) / s)

    def dot(u, v):
        return (u * v).sum(dim=axes, keepdim=True)

    x, r = torch.zeros_like(b), b.clone()
    z = precondition(r)
    p, rz = z.clone(), dot(r, z)
    rz0 = rz.clone()
    for it in range(600):
        q = matvec(p)
        alpha = rz / dot(p, q).clamp_min(1e-300)
        x, r = x + alpha * p, r - alpha * q
        z = precondition(r)
        new = dot(r, z)
        p, rz = z + (new / rz.clamp_min(1e-300)) * p, new
        if it % 10 == 9 and float((rz / rz0).max()) < 1e-28:
            break
    return x


def _gelu_net(p, X, Phi, Psi, layers):
    """The spectral neural operator on (B, P, CIN) inputs, channels last."""
    U = X @ p["W_lift"].T + p["b_lift"]
    for l in range(layers):
        hat = Phi @ U
        mixed = torch.einsum("qij,bqj->bqi", p[f"R{l}"], hat)
        U = Psi @ mixed + U @ p[f"W{l}"].T + p[f"b{l}"]
        if l < layers - 1:
            U = torch.nn.functional.gelu(U)
    Q = torch.nn.functional.gelu(U @ p["W_p1"].T + p["b_p1"])
    return (Q @ p["W_p2"].T + p["b_p2"])[..., 0]


def _train_exact(case, seed):
    model, x, target = _train_inputs(case, seed)
    n, m, B = case["n"], case["modes"], case["batch"]
    V = _vander("legendre", n, n)
    w = _nodes("legendre", n)[1]
    F = ((V * w[:, None]).T * (np.arange(n) + 0.5)[:, None])[:m]
    Phi, Psi = _dev(np.kron(F, F)), _dev(np.kron(V[:, :m], V[:, :m]))
    p = {k: v.detach().double().requires_grad_(True) for k, v in model.params.items()}
    pred = _gelu_net(p, x.double().reshape(B, n * n, CIN), Phi, Psi, model.cfg.layers)
    loss = 0.5 * (pred - target.double().reshape(B, n * n)).square().mean()
    loss.backward()
    grads = {k: v.grad.detach() for k, v in p.items()}
    # Adam's first step divides every gradient by its own size: no exact value
    return {"loss": float(loss.detach()), "grads": grads, "params": {k: None for k in p}}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "helmholtz":
        Ns, alphas = _helmholtz_plan(case["count"], case["top"], case["plan"])
        b, out, at = _helmholtz_rhs(case, seed), [], 0
        for N in sorted(set(Ns.tolist())):
            idx = np.nonzero(Ns == N)[0]
            size = len(idx) * (N - 2) ** 2
            rhs = b[at:at + size].reshape(len(idx), N - 2, N - 2)
            out.append(_helmholtz_solve(case["family"], N, 2, alphas[idx] ** 2, rhs).reshape(-1))
            at += size
        return torch.cat(out)
    nd, N = case["ndim"], case["N"]
    if kind == "poisson":
        f = prepare(case, seed)["f"]
        b = _kron([_dev(_scalar_product(case["family"], N))] * nd, f)
        c = _helmholtz_solve(case["family"], N, nd, case["alpha2"], b)
        return c, _kron([_dev(_dirichlet(_vander(case["family"], N, N)))] * nd, c)
    if kind == "roundtrip":
        c = _roundtrip_input(case, seed).double()
        V = _vander(case["family"], N, N)
        if case["precision"] != "lifted":
            return _kron([_dev(V)] * nd, c), c
        # values LIFT_LEFT and LIFT_RIGHT at x = -1 and 1, projected in y
        B = _dirichlet(V)
        M = _galerkin(case["family"], N)[0]
        proj = np.linalg.solve(M, _scalar_product(case["family"], N) @ np.ones(N))
        x = V[:, 1]
        left, right = LIFT_LEFT * 0.5 * (1.0 - x), LIFT_RIGHT * 0.5 * (1.0 + x)
        u = _kron([_dev(B)] * 2, c) + _dev(np.outer(left + right, B @ proj))
        return u, c
    if kind == "operator":
        matvec, _ = _varcoef(case, seed)
        return matvec(prepare(case, seed)["u"])
    if kind == "mixed" and nd == 3 and case["batch"] * N**4 > 8 * 128**4:
        return None
    return _varcoef_solve(case, seed)
