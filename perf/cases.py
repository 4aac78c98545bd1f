"""The library's work as its users call it, for timing and comparing builds.

Every case is one pass through the public entry points (``compile_osqp`` and its
engine, ``solve_classes``, ``compile_qdldl_variant``, ``QuadrotorSQP``) on the MPC
classes of ``warpmpc_b200.problems`` at some horizon, with float32 data resident on
the GPU.  Kinds of case:

* ``solve``     P, A, q, l, u of every instance are new: factor + 25 ADMM iterations,
                warm-started (a controller that runs every sample) or cold;
* ``shared``    one P and A for the whole batch, factored beforehand
                (linear time-invariant plants: ``solve_with_factor_warm_start``);
* ``mixed``     four problem classes in one launch with termination checks;
* ``gradient``  a differentiable solve and its backward pass (learning through MPC);
* ``adaptive``  per-instance rho adaptation;
* ``factor``    ``compile_qdldl_variant(...).factor`` and ``.solve`` on new KKT values;
* ``linsolve``  ``.solve`` alone on a kept factorization;
* ``sqp``       one real-time iteration of the nonlinear quadrotor SQP: linearise at the
                current trajectory and solve the QP.

Inputs are drawn on the GPU from the seed with the distributions of
``problems.draw_params``; plans come from one fixed representative instance per class,
as the reference builds its scaling from representative values, and are kept.
"""

from __future__ import annotations

import functools

import numpy as np
import torch

from warpmpc_b200 import problems, quadrotor_sqp
from warpmpc_b200.jax_osqp import OSQPSettings, compile_osqp, solve_classes
from warpmpc_b200.jax_qdldl import compile_qdldl_variant

# (states, inputs, state box, input box, x0 range, dynamics) of the library's MPC classes
_CLASSES = {
    "small": (4, 2, 5.0, 1.0, 2.0, "small"),
    "cartpole": (4, 1, 5.0, 10.0, 2.0, "small"),
    "quadrotor": (12, 4, 10.0, 2.0, 1.0, "quadrotor"),
}
_MIXED = (("small", 10), ("small", 40), ("quadrotor", 20), ("quadrotor", 30))


def listed():
    return [
        # one robot's controller: the smallest call, latency is all that counts
        dict(name="quadrotor_1", kind="solve", plant="quadrotor", horizon=30, batch=1, warm=True),
        # a few candidate plans or a small fleet, an odd count
        dict(name="cartpole_97_cold", kind="solve", plant="cartpole", horizon=50, batch=97, warm=False),
        # sampling-based evaluation or reinforcement learning with an MPC layer, ordinary size
        dict(name="quadrotor_1000", kind="solve", plant="quadrotor", horizon=30, batch=1000, warm=True),
        # the benchmark's closed-loop step, the largest call
        dict(name="quadrotor_65536", kind="solve", plant="quadrotor", horizon=30, batch=65536, warm=True),
        # the small pattern at the benchmark's batch
        dict(name="small_65536_cold", kind="solve", plant="small", horizon=10, batch=65536, warm=False),
        # a heterogeneous fleet with early exit
        dict(name="mixed_4x4000", kind="mixed", batch=4000),
        # identical plants: one factorization for all, only the vectors change
        dict(name="shared_quadrotor_8192", kind="shared", plant="quadrotor", horizon=30, batch=8192),
        # learning through the controller: solve and backward
        dict(name="gradient_cartpole_16384", kind="gradient", plant="cartpole", horizon=50, batch=16384),
        # badly scaled instances: rho adapts per instance
        dict(name="adaptive_quadrotor_2000", kind="adaptive", plant="quadrotor", horizon=20, batch=2000),
        # the linear-algebra layer alone: factor and solve, then solves on a kept factor
        dict(name="factor_quadrotor_4097", kind="factor", plant="quadrotor", horizon=30, batch=4097),
        dict(name="linsolve_quadrotor_20000", kind="linsolve", plant="quadrotor", horizon=30, batch=20000),
        # nonlinear MPC, one real-time iteration for a fleet
        dict(name="sqp_quadrotor_5000", kind="sqp", horizon=40, batch=5000),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "mixed", "shared", "gradient", "adaptive", "factor",
                       "linsolve", "sqp"])
    def size(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    if kind == "mixed":
        return dict(kind=kind, batch=size(100, 8000))
    if kind == "sqp":
        return dict(kind=kind, horizon=rng.choice([20, 40]), batch=size(100, 8000))
    plant = rng.choice(["small", "cartpole", "quadrotor"])
    horizon = rng.choice([10, 15, 20, 30]) if plant == "quadrotor" else rng.choice([10, 20, 40, 50])
    case = dict(kind=kind, plant=plant, horizon=horizon)
    if kind == "solve":
        case.update(batch=size(1, 65000), warm=rng.random() < 0.5)
    elif kind in ("shared", "gradient"):
        case.update(batch=size(10, 16000))
    elif kind == "adaptive":
        case.update(batch=size(10, 8000))
    else:
        case.update(batch=size(10, 32000))
    return case


# ---------------------------------------------------------------------------
# what a user's program keeps: plans and compiled solvers, one per pattern
# ---------------------------------------------------------------------------

def _mpc_class(plant, horizon):
    nx, nu, x_max, u_max, x0_max, dyn = _CLASSES[plant]
    return problems.MPCClass(f"{plant}-n{horizon}", nx, nu, horizon, x_max, u_max, x0_max, dyn)


def _settings(kind):
    s = dict(problems.DEFAULT_SETTINGS)
    if kind == "mixed":
        s.update(max_iter=50, check_termination=1, eps_abs=1e-3, eps_rel=0.0)
    elif kind == "adaptive":
        s.update(max_iter=60, adaptive_rho=True, adaptive_rho_interval=10)
    return OSQPSettings(**s)


@functools.lru_cache(maxsize=None)
def _plan(plant, horizon, kind):
    cls = _mpc_class(plant, horizon)
    return problems.make_plan(problems.make_batch(cls, 1, seed=0), _settings(kind))


@functools.lru_cache(maxsize=None)
def _compiled(plant, horizon, kind):
    return compile_osqp(_plan(plant, horizon, kind), np.float32, qdldl_backend="cuda", transpose_work=True,
                        derivatives=kind == "gradient")


@functools.lru_cache(maxsize=None)
def _qdldl(plant, horizon):
    return compile_qdldl_variant(_plan(plant, horizon, "solve").qdldl_plan, np.float32, backend="cuda",
                                 transpose_work=True)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _draws(cls, batch, gen):
    """``problems.draw_params``'s distributions, drawn on the GPU in float32."""
    nx, nu = cls.nx, cls.nu
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    uniform = lambda lo, hi, *s: lo + (hi - lo) * torch.rand(*s, generator=gen, device="cuda")  # noqa: E731
    eye = torch.eye(nx, device="cuda")
    if cls.kind == "quadrotor":
        mask = torch.zeros(nx, nx, device="cuda")
        for bi, bj in ((0, 2), (2, 1), (1, 3), (2, 2), (3, 3)):
            mask[3 * bi : 3 * bi + 3, 3 * bj : 3 * bj + 3] = 1.0
        a = eye + 0.02 * 0.3 * normal(batch, nx, nx) * mask
        b = 0.5 * normal(batch, nx, nu)
    else:
        a = eye + 0.1 * normal(batch, nx, nx)
        radius = np.max(np.abs(np.linalg.eigvals(a.cpu().numpy())), axis=1)
        a = a * torch.from_numpy(np.minimum(1.0, 1.02 / radius).astype(np.float32)).cuda()[:, None, None]
        b = 0.1 * normal(batch, nx, nu)
    return problems.MPCParams(cls, a, b, uniform(1.0, 10.0, batch, nx), uniform(0.1, 1.0, batch, nu),
                              uniform(-cls.x0_max, cls.x0_max, batch, nx), uniform(-0.5, 0.5, batch, nx))


def _inputs(plant, horizon, batch, seed, warm=True, shared=False):
    """P, A, q, l, u and a warm start: the plan of the plant coasting from x0
    (no input), its constraint values inside the bounds, small multipliers."""
    cls = _mpc_class(plant, horizon)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    params = _draws(cls, batch, gen)
    if shared:  # one plant: every instance has the first one's dynamics and weights
        for f in ("a", "b", "qd", "rd"):
            v = getattr(params, f)
            setattr(params, f, v[:1].expand_as(v).contiguous())
    p, a, q, l, u = (t.float().contiguous() for t in problems.qp_from_params(params))
    if shared:
        p, a = p[:1].contiguous(), a[:1].contiguous()
    if not warm:
        return p, a, q, l, u, None
    x, states = params.x0, []
    for _ in range(cls.horizon + 1):
        states.append(x)
        x = torch.bmm(params.a, x[:, :, None])[:, :, 0].clamp(-cls.x_max, cls.x_max)
    wx = torch.cat(states + [torch.zeros(batch, cls.horizon * cls.nu, device="cuda")], 1)
    n_eq = (cls.horizon + 1) * cls.nx
    wz = torch.cat([l[:, :n_eq], torch.minimum(torch.maximum(wx, l[:, n_eq:]), u[:, n_eq:])], 1)
    wy = 0.01 * torch.randn(batch, l.shape[1], generator=gen, device="cuda")
    wy[:, n_eq:] = 0.0
    return p, a, q, l, u, (wx.contiguous(), wz.contiguous(), wy)


def _kkt_values(plant, horizon, batch, seed):
    """(nnz_kkt, batch) KKT values of the instances' scaled QPs."""
    plan = _plan(plant, horizon, "solve")
    p, a, *_ = _inputs(plant, horizon, batch, seed, warm=False)
    f = lambda v: torch.as_tensor(np.asarray(v), dtype=torch.float32, device="cuda")  # noqa: E731
    ix = lambda v: torch.as_tensor(np.asarray(v), dtype=torch.int64, device="cuda")  # noqa: E731
    vals = f(plan.kkt_upper.data)[:, None].repeat(1, batch)
    vals[ix(plan.p_to_kkt)] = (p * f(plan.p_scale) + f(plan.p_diag_sigma)).T
    vals[ix(plan.a_to_kkt)] = (a * f(plan.a_scale)).T
    rhs = torch.randn(plan.qdldl_plan.n, batch, generator=torch.Generator(device="cuda").manual_seed(seed + 1),
                      device="cuda")
    return vals, rhs


def prepare(case, seed):
    kind, batch = case["kind"], case["batch"]
    if kind == "sqp":
        sqp = quadrotor_sqp.QuadrotorSQP(case["horizon"], quadrotor_sqp.make_data(batch, seed), "cuda", iterations=1)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        z = quadrotor_sqp.initial_guess(sqp.plan, sqp.x0)
        z = z + 0.01 * torch.randn(z.shape, generator=gen, device="cuda")
        m = int(sqp.plan.constraint_offsets[-1])
        warm = (torch.zeros_like(z), torch.zeros(batch, m, device="cuda"), torch.zeros(batch, m, device="cuda"))
        return dict(kind=kind, sqp=sqp, z=z, warm=warm)
    if kind == "mixed":
        work = []
        for i, (plant, horizon) in enumerate(_MIXED):
            *qp, warm = _inputs(plant, horizon, batch, seed * 4 + i)
            work.append((_compiled(plant, horizon, "mixed").engine, *qp, warm))
        return dict(kind=kind, work=work)
    plant, horizon = case["plant"], case["horizon"]
    if kind in ("factor", "linsolve"):
        q = _qdldl(plant, horizon)
        vals, rhs = _kkt_values(plant, horizon, batch, seed)
        if kind == "factor":
            return dict(kind=kind, qdldl=q, values=vals, rhs=rhs)
        lx, _, dinv = q.factor(vals)
        return dict(kind=kind, qdldl=q, lx=lx, dinv=dinv, rhs=rhs)
    c = _compiled(plant, horizon, kind)
    if kind == "shared":
        p, a, q, l, u, warm = _inputs(plant, horizon, batch, seed, shared=True)
        lx, dinv = c.factor(p, a)
        return dict(kind=kind, solver=c, args=(lx, dinv, p, a, q, l, u, *warm))
    p, a, q, l, u, warm = _inputs(plant, horizon, batch, seed, warm=kind == "solve" and case["warm"])
    if kind == "gradient":
        cx = torch.randn(q.shape, generator=torch.Generator(device="cuda").manual_seed(seed + 1), device="cuda")
        return dict(kind=kind, solver=c, args=(p, a, q, l, u), cx=cx)
    return dict(kind=kind, solver=c, args=(p, a, q, l, u) if warm is None else (p, a, q, l, u, *warm))


def run(state):
    kind = state["kind"]
    if kind == "sqp":
        s = state["sqp"]
        r = s.sqp.solve_qp(state["z"], s.x0, state["warm"])
        return (r.direction, r.z, r.y)
    if kind == "mixed":
        return [list(o) for o in solve_classes(state["work"])]
    if kind == "factor":
        x, lx, d = state["qdldl"].factor_and_solve(state["values"], state["rhs"])
        return (x, lx, d)
    if kind == "linsolve":
        return state["qdldl"].solve(state["lx"], state["dinv"], state["rhs"])
    c = state["solver"]
    if kind == "shared":
        return c.solve_with_factor_warm_start(*state["args"])
    if kind == "gradient":
        args = [t.detach().requires_grad_(True) for t in state["args"]]
        x, y = c.solve_xy(*args)
        return (x.detach(), y.detach(), *torch.autograd.grad(x, args, state["cx"]))
    if kind == "adaptive":
        out = c.solve(*state["args"])
        return (*out, c.engine.last_rho, c.engine.last_rho_updates)
    return c.solve_warm_start(*state["args"]) if len(state["args"]) == 8 else c.solve(*state["args"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _work_qp(plan, batch, iters, shared=False, warm=True):
    """Inputs and outputs once; one factorization per instance (unless shared) and iters KKT solves."""
    k = plan.qdldl_plan
    cols = np.diff(np.asarray(k.lp)[: k.n + 1])
    fac = float(np.sum(cols * (cols + 1) + cols))
    vec = 3 * (plan.n + 2 * plan.m) if warm else 2 * (plan.n + 2 * plan.m)
    data = (0 if shared else plan.nnz_p + plan.nnz_a) + vec
    return 4.0 * batch * data, batch * ((0.0 if shared else fac) + iters * (4.0 * k.nnz_l + 12.0 * k.n))


def work(case):
    kind, batch = case["kind"], case["batch"]
    if kind == "sqp":
        n, m, nnz_a, nnz_l = 16 * case["horizon"] + 12, 12 + 16 * case["horizon"], 142 * case["horizon"] + 12, 0
        nnz_l = 8 * (n + m)
        return {"bytes": 4.0 * batch * (6 * n + 6 * m), "flops": batch * (100.0 * nnz_a + 25 * (4.0 * nnz_l + 12.0 * (n + m)))}
    if kind == "mixed":  # early exit: at least one iteration each
        parts = [_work_qp(_plan(p, h, kind), batch, 1) for p, h in _MIXED]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    plan = _plan(case["plant"], case["horizon"], kind if kind in ("adaptive", "gradient") else "solve")
    k = plan.qdldl_plan
    if kind in ("factor", "linsolve"):
        _, fac = _work_qp(plan, batch, 0)
        if kind == "factor":
            return {"bytes": 4.0 * batch * (k.nnz_a + k.nnz_l + 3 * k.n), "flops": fac + batch * 4.0 * k.nnz_l}
        return {"bytes": 4.0 * batch * (k.nnz_l + 3 * k.n), "flops": batch * 4.0 * k.nnz_l}
    iters = 60 if kind == "adaptive" else 25
    nbytes, flops = _work_qp(plan, batch, 2 * iters if kind == "gradient" else iters, shared=kind == "shared",
                             warm=kind == "shared" or bool(case.get("warm")))
    if kind == "gradient":
        nbytes += 4.0 * batch * (2 * plan.n + 2 * plan.m + plan.nnz_p + plan.nnz_a)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain NumPy and torch
# ---------------------------------------------------------------------------

class _Ldl64:
    """Sparse L D L^T of a batch of quasi-definite matrices in float64, column
    by column (right-looking), for one pattern and elimination order."""

    def __init__(self, n, rows, cols, perm):
        inv = np.empty(n, dtype=np.int64)
        inv[np.asarray(perm)] = np.arange(n)
        self.n, self.perm = n, torch.as_tensor(np.asarray(perm, dtype=np.int64), device="cuda")
        pr, pc = inv[rows], inv[cols]
        struct = [set() for _ in range(n)]
        for r, c in zip(np.maximum(pr, pc), np.minimum(pr, pc)):
            if r != c:
                struct[c].add(int(r))
        self.cols = []
        for c in range(n):
            s = sorted(struct[c])
            self.cols.append(s)
            if s:
                struct[s[0]].update(s[1:])
        self.slot = {(c, c): c for c in range(n)}
        for c in range(n):
            for r in self.cols[c]:
                self.slot[(r, c)] = len(self.slot)
        ix = lambda v: torch.as_tensor(np.asarray(v, dtype=np.int64), device="cuda")  # noqa: E731
        self.input = ix([self.slot[(max(r, c), min(r, c))] for r, c in zip(pr, pc)])
        self.l_slots = [ix([self.slot[(r, c)] for r in self.cols[c]]) for c in range(n)]
        self.l_rows = [ix(self.cols[c]) for c in range(n)]
        self.updates = []
        for c in range(n):
            s = self.cols[c]
            pairs = [(i, j) for j in range(len(s)) for i in range(j, len(s))]
            self.updates.append((ix([self.slot[(s[i], s[j])] for i, j in pairs]), ix([i for i, _ in pairs]),
                                 ix([j for _, j in pairs])))

    def factor(self, values):
        w = torch.zeros(len(self.slot), values.shape[1], dtype=torch.float64, device="cuda")
        w.index_add_(0, self.input, values)
        for c in range(self.n):
            if not self.cols[c]:
                continue
            y = w[self.l_slots[c]]
            l = y / w[c]
            dst, i, j = self.updates[c]
            w[dst] -= l[i] * y[j]
            w[self.l_slots[c]] = l
        self.w = w
        return self

    def solve(self, rhs):
        x = rhs[self.perm]
        for c in range(self.n):
            if self.cols[c]:
                x[self.l_rows[c]] -= self.w[self.l_slots[c]] * x[c]
        x /= self.w[: self.n]
        for c in reversed(range(self.n)):
            if self.cols[c]:
                x[c] -= (self.w[self.l_slots[c]] * x[self.l_rows[c]]).sum(0)
        out = torch.empty_like(x)
        out[self.perm] = x
        return out


def _ruiz(prows, pcols, pvals, arows, acols, avals, q, m, rounds):
    """OSQP's equilibration of one representative problem (P by its upper triangle)."""
    n = q.size
    pv, av, qv = pvals.copy(), avals.copy(), q.copy()
    d, e, c = np.ones(n), np.ones(m), 1.0

    def clip(v):
        v = np.asarray(v, dtype=np.float64)
        return np.where(v < 1e-4, 1.0, np.minimum(v, 1e4))

    def colmax(vals, idx, size):
        out = np.zeros(size)
        np.maximum.at(out, idx, np.abs(vals))
        return out

    for _ in range(rounds):
        ds = 1.0 / np.sqrt(clip(np.maximum(colmax(pv, pcols, n), colmax(av, acols, n))))
        es = 1.0 / np.sqrt(clip(colmax(av, arows, m)))
        pv *= ds[prows] * ds[pcols]
        av *= es[arows] * ds[acols]
        qv *= ds
        d *= ds
        e *= es
        g = 1.0 / float(clip(max(float(np.mean(colmax(pv, pcols, n))), float(clip(np.max(np.abs(qv)))))))
        pv *= g
        qv *= g
        c *= g
    return d, e, c


@functools.lru_cache(maxsize=2)
def _reference(plant, horizon):
    """Pattern, scaling, rho and elimination of a class in 64 bits."""
    cls = _mpc_class(plant, horizon)
    rep = problems.make_batch(cls, 1, seed=0)
    pu, am = rep.p_matrix0.tocoo(), rep.a_matrix0.tocoo()  # CSC entry order
    prows, pcols, arows, acols = (np.asarray(v, dtype=np.int64) for v in (pu.row, pu.col, am.row, am.col))
    n, m = pu.shape[0], am.shape[0]
    d, e, c = _ruiz(prows, pcols, pu.data.astype(np.float64), arows, acols, am.data.astype(np.float64),
                    rep.q[0].astype(np.float64), m, 10)
    equality = np.abs(e * (rep.u[0].astype(np.float64) - rep.l[0].astype(np.float64))) < 1e-4
    rho = np.where(equality, 1e3 * 0.1, 0.1)
    rows = np.concatenate([prows, acols, n + np.arange(m)])
    cols = np.concatenate([pcols, n + arows, n + np.arange(m)])
    ldl = _Ldl64(n + m, rows, cols, _plan(plant, horizon, "solve").qdldl_plan.p)
    return prows, pcols, arows, acols, n, m, d, e, c, rho, ldl


def _exact_qp(plant, horizon, p, a, q, l, u, warm, iters=25):
    prows, pcols, arows, acols, n, m, d, e, c, rho, ldl = _reference(plant, horizon)
    f = lambda v: torch.as_tensor(np.asarray(v, dtype=np.float64), device="cuda")[:, None]  # noqa: E731
    p, a, q, l, u = (t.double().T for t in (p, a, q, l, u))
    batch, sigma, alpha = q.shape[1], 1e-6, 1.6
    ps = p * f(c * d[prows] * d[pcols]) + f(np.where(prows == pcols, sigma, 0.0))
    ks = torch.cat([ps, a * f(e[arows] * d[acols]), -1.0 / f(rho).expand(m, ps.shape[1])])
    ldl.factor(ks)
    qs, ls, us, rv = q * f(c * d), l * f(e), u * f(e), f(rho)
    if warm is None:
        x, z, y = (torch.zeros(k, batch, dtype=torch.float64, device="cuda") for k in (n, m, m))
    else:
        x, z, y = warm[0].double().T / f(d), warm[1].double().T * f(e), warm[2].double().T * f(c / e)
    for _ in range(iters):
        sol = ldl.solve(torch.cat([sigma * x - qs, z - y / rv]))
        zt = z + (sol[n:] - y) / rv
        zr = alpha * zt + (1 - alpha) * z
        x = alpha * sol[:n] + (1 - alpha) * x
        z = torch.minimum(torch.maximum(zr + y / rv, ls), us)
        y = y + rv * (zr - z)
    x, z, y = x * f(d), z / f(e), y * f(e / c)
    # the residuals of a float32 iterate near convergence are its own rounding, not the 64-bit run's;
    # the classes' P is diagonal
    return (x.T, z.T, y.T, None, None, (x * (0.5 * (p * x) + q)).sum(0))


def exact(case, seed):
    """64-bit results: None for cases whose path is decided by comparisons of
    iterates (early exit, rho adaptation), for the derivative of an iterate
    that has not converged (its active set is such a decision too), and for
    the nonlinear model's linearisation."""
    kind, batch = case["kind"], case["batch"]
    if kind in ("mixed", "adaptive", "sqp"):
        return None
    plant, horizon = case["plant"], case["horizon"]
    if kind in ("factor", "linsolve"):
        plan = _plan(plant, horizon, "solve")
        vals, rhs = _kkt_values(plant, horizon, batch, seed)
        k = plan.kkt_upper.tocoo()
        ldl = _Ldl64(plan.qdldl_plan.n, np.asarray(k.row, np.int64), np.asarray(k.col, np.int64), plan.qdldl_plan.p)
        ldl.factor(vals.double())
        x = ldl.solve(rhs.double())
        if kind == "linsolve":
            return x
        lx = torch.cat([ldl.w[s] for s in ldl.l_slots if s.numel()])
        return (x, lx, ldl.w[: ldl.n])
    p, a, q, l, u, warm = _inputs(plant, horizon, batch, seed, warm=kind == "shared" or bool(case.get("warm")),
                                  shared=kind == "shared")
    out = _exact_qp(plant, horizon, p, a, q, l, u, warm)
    if kind == "gradient":
        return (out[0], out[2], None, None, None, None, None)
    return out
