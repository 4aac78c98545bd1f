"""The band form of the persistent solve on the GPU (warpmpc_b200/csrc/band.cu).

The arithmetic and its order are the other forms': iterates equal the float32
oracle's bit for bit, and checked or rho-adapting solves equal the streaming
form's, iteration and refactorization counts included.  ``WMPC_STREAM_BAND=1``
runs it wherever its tables can be built, 0 nowhere.
"""

import numpy as np
import pytest

from oracle import osqp_ref
from warpmpc_b200 import native, problems
from warpmpc_b200.jax_osqp import OSQPSettings, compile_osqp, solve_classes

pytestmark = pytest.mark.gpu


def _dev(*arrays):
    import torch

    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _compile(monkeypatch, plan, band):
    monkeypatch.setenv("WMPC_STREAM_BAND", str(band))
    comp = compile_osqp(plan, np.float32, qdldl_backend="cuda", transpose_work=True, mode="persistent")
    monkeypatch.delenv("WMPC_STREAM_BAND")
    return comp


def _warm(plan, batch, seed):
    rng = np.random.default_rng(seed)
    return [(rng.standard_normal((batch, k)) * 0.1).astype(np.float32) for k in (plan.n, plan.m, plan.m)]


SHORT = problems.MPCClass("short quadrotor", 12, 4, 2, 10.0, 2.0, 1.0, "quadrotor")


@pytest.mark.parametrize("cls,batch,ctas", [(problems.SMALL, 1, 1), (problems.SMALL, 9500, 2), (problems.CARTPOLE, 97, 1),
                                            (problems.CARTPOLE, 4801, 1), (SHORT, 33, 1), (problems.QUADROTOR, 32, 1),
                                            (problems.QUADROTOR, 4801, 1)], ids=lambda v: getattr(v, "name", str(v)))
def test_band_form_bitexact(cuda_device, monkeypatch, cls, batch, ctas):
    """One lane, whole and partial tiles, one and two CTAs per SM, 8- and
    16-row windows, a chain of a few chunks, several tiles per CTA."""
    from oracle.cpu_baseline import CpuOSQP

    b = problems.make_batch(cls, batch, seed=31)
    plan = problems.make_plan(b)
    comp = _compile(monkeypatch, plan, 1)
    got = comp.engine.solve(*_dev(b.p_values, b.a_values, b.q, b.l, b.u))
    launch = native.stream_last_launch()
    assert launch["form"] == "band" and launch["ctas_per_sm"] == ctas, launch
    ref = CpuOSQP(plan).solve(b.p_values, b.a_values, b.q, b.l, b.u)
    for name, g, r in zip(("x", "z", "y"), got[:3], ref[:3]):
        np.testing.assert_array_equal(g.cpu().numpy(), r, err_msg=name)
    assert not np.any(comp.engine.last_status.cpu().numpy() & 8)


@pytest.mark.parametrize("cls", [problems.SMALL, problems.QUADROTOR], ids=lambda c: c.name)
def test_band_form_warm_start_shared_matrices(cuda_device, monkeypatch, cls):
    b = problems.make_batch(cls, 45, seed=6)
    plan = problems.make_plan(b)
    comp = _compile(monkeypatch, plan, 1)
    warm = _warm(plan, 45, 2)
    args = (b.p_values[:1], b.a_values[:1], b.q, b.l, b.u)
    got = comp.engine.solve(*_dev(*args), warm=tuple(_dev(*warm)))
    ref = osqp_ref.solve_warm_start(plan, *args, *warm)
    for g, r in zip(got[:3], ref[:3]):
        np.testing.assert_array_equal(g.cpu().numpy(), r)


@pytest.mark.parametrize("cls,batch", [(problems.SMALL, 40), (problems.SMALL, 9500), (problems.CARTPOLE, 5300),
                                       (problems.QUADROTOR, 70)], ids=lambda v: getattr(v, "name", str(v)))
def test_band_form_termination_checks(cuda_device, monkeypatch, cls, batch):
    """Tiles that stop early, and what follows them on the same CTA."""
    b = problems.make_batch(cls, batch, seed=3)
    plan = problems.make_plan(b, OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 60}))
    band, plain = _compile(monkeypatch, plan, 1), _compile(monkeypatch, plan, 0)
    args = _dev(b.p_values, b.a_values, b.q, b.l, b.u)
    for warm in (None, tuple(_dev(*_warm(plan, batch, 8)))):
        got = band.engine.solve(*args, warm=warm, check_termination=5)
        assert native.stream_last_launch()["form"] == "band"
        want = plain.engine.solve(*args, warm=warm, check_termination=5)
        assert native.stream_last_launch()["form"] != "band"
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())
        iters = band.engine.last_iters.cpu().numpy()
        np.testing.assert_array_equal(iters, plain.engine.last_iters.cpu().numpy())
        np.testing.assert_array_equal(band.engine.last_status.cpu().numpy(), plain.engine.last_status.cpu().numpy())


@pytest.mark.parametrize("cls,batch", [(problems.SMALL, 75), (problems.CARTPOLE, 5000)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_band_form_adaptive_rho(cuda_device, monkeypatch, cls, batch):
    b = problems.make_batch(cls, batch, seed=37)
    settings = OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 30, "adaptive_rho": True,
                               "adaptive_rho_interval": 8, "adaptive_rho_tolerance": 2.0})
    plan = problems.make_plan(b, settings)
    band, plain = _compile(monkeypatch, plan, 1), _compile(monkeypatch, plan, 0)
    args = _dev(b.p_values, b.a_values, b.q, b.l, b.u)
    got, want = band.engine.solve(*args), plain.engine.solve(*args)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())
    upd = band.engine.last_rho_updates.cpu().numpy()
    np.testing.assert_array_equal(upd, plain.engine.last_rho_updates.cpu().numpy())
    assert upd.sum() > 0


@pytest.mark.parametrize("check", [0, 5])
def test_band_form_classes(cuda_device, monkeypatch, check):
    """Classes of both window widths in one launch, several tiles per CTA."""
    specs = [(problems.QUADROTOR, 2000), (problems.SMALL, 3001), (problems.CARTPOLE, 1500)]
    items = {0: [], 1: []}
    for k, (cls, batch) in enumerate(specs):
        b = problems.make_batch(cls, batch, seed=20 + k)
        plan = problems.make_plan(b, OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 30}))
        for f in (0, 1):
            items[f].append((_compile(monkeypatch, plan, f).engine, *_dev(b.p_values, b.a_values, b.q, b.l, b.u), None))
    got = solve_classes(items[1], check_termination=check)
    assert native.stream_last_launch()["form"] == "band"
    want = solve_classes(items[0], check_termination=check)
    for gs, ws in zip(got, want):
        for g, w in zip(gs, ws):
            np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())


def test_band_form_beside_a_tuned_class(cuda_device, monkeypatch):
    """A class compiled with schedule knobs runs them alone; in a launch whose other
    classes hold most of the work it runs the band form with them."""
    specs, work, alone = [(problems.QUADROTOR, 500), (problems.SMALL, 700)], [], []
    for k, (cls, batch) in enumerate(specs):
        b = problems.make_batch(cls, batch, seed=40 + k)
        with monkeypatch.context() as m:
            if cls is problems.SMALL:
                m.setenv("WMPC_STREAM_FRONTIER_COPIES", "1")
            comp = compile_osqp(problems.make_plan(b), np.float32, qdldl_backend="cuda", transpose_work=True)
        args = _dev(b.p_values, b.a_values, b.q, b.l, b.u)
        alone.append([o.clone() for o in comp.engine.solve(*args)])
        form = native.stream_last_launch()["form"]
        assert (form == "band") == (cls is problems.QUADROTOR)
        work.append((comp.engine, *args, None))
    outs = solve_classes(work)
    assert native.stream_last_launch()["form"] == "band"
    for out, want in zip(outs, alone):
        for g, w in zip(out[:3], want[:3]):
            np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())
    solve_classes(work[1:])
    assert native.stream_last_launch()["form"] != "band"


def test_band_form_choice(cuda_device):
    """Which form a solve runs by default: long chains the band form, others
    the streaming forms where one tile per SM does not bound them."""
    for cls, batch, band in ((problems.QUADROTOR, 40, True), (problems.CARTPOLE, 5000, True), (problems.SMALL, 40, False)):
        b = problems.make_batch(cls, batch, seed=1)
        comp = compile_osqp(problems.make_plan(b), np.float32, qdldl_backend="cuda", transpose_work=True)
        comp.engine.solve(*_dev(b.p_values, b.a_values, b.q, b.l, b.u))
        assert (native.stream_last_launch()["form"] == "band") == band, cls.name


@pytest.mark.parametrize("kind,nx,nu,horizon,limit", [
    ("small", 4, 2, 2, 0), ("small", 4, 1, 6, 0), ("small", 2, 1, 15, 0), ("small", 5, 1, 6, 0),  # short chains
    ("quadrotor", 12, 4, 1, 148), ("small", 4, 1, 10, 148), ("small", 5, 1, 20, 148), ("small", 2, 1, 50, 148),
    ("quadrotor", 12, 4, 10, 148), ("small", 4, 1, 20, None), ("quadrotor", 12, 4, 15, None)])
def test_band_form_choice_by_chain(cuda_device, kind, nx, nu, horizon, limit):
    """Up to how many tiles a pattern runs the band form by default: none for a short
    chain, one per SM, or any number."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cls = problems.MPCClass("x", nx, nu, horizon, 5.0, 5.0, 1.0, kind)
    b = problems.make_batch(cls, 2, seed=1)
    comp = compile_osqp(problems.make_plan(b), np.float32, qdldl_backend="cuda", transpose_work=True)
    args = _dev(b.p_values, b.a_values, b.q, b.l, b.u)
    for tiles in (1, sms, sms + 1):
        comp.engine.solve(*[t.repeat(tiles * 16, 1) for t in args], max_iter=2)
        band = native.stream_last_launch()["form"] == "band"
        assert band == (limit is None or (limit > 0 and tiles <= sms)), tiles
    comp.engine.solve(*[t.repeat((sms + 1) * 16, 1) for t in args], max_iter=2, check_termination=1)
    band = native.stream_last_launch()["form"] == "band"
    assert band == (limit is None and (kind, horizon) != ("small", 20))


def test_band_form_wait_timeout(cuda_device, monkeypatch):
    """Waits limited to one microsecond give up: every instance is marked, the
    launch returns, and the next solve is right."""
    import torch

    b = problems.make_batch(problems.CARTPOLE, 96, seed=5)
    plan = problems.make_plan(b)
    comp = _compile(monkeypatch, plan, 1)
    args = _dev(b.p_values, b.a_values, b.q, b.l, b.u)
    monkeypatch.setenv("WMPC_STREAM_WAIT_LIMIT_NS", "1000")
    comp.engine.solve(*args)
    torch.cuda.synchronize()
    assert native.stream_last_launch()["form"] == "band"
    status = comp.engine.last_status.cpu().numpy()
    assert np.all(status & native.STATUS_KERNEL_ABORT), np.unique(status)
    monkeypatch.delenv("WMPC_STREAM_WAIT_LIMIT_NS")
    got = comp.engine.solve(*args)
    assert not np.any(comp.engine.last_status.cpu().numpy() & native.STATUS_KERNEL_ABORT)
    ref = osqp_ref.solve(plan, b.p_values, b.a_values, b.q, b.l, b.u)
    for g, r in zip(got[:3], ref[:3]):
        np.testing.assert_array_equal(g.cpu().numpy(), r)


@pytest.mark.parametrize("band", [0, 1], ids=["stream", "band"])
@pytest.mark.parametrize("cls,batch,shared", [(problems.SMALL, 37, True), (problems.CARTPOLE, 96, False),
                                              (problems.SMALL, 1, False), (problems.QUADROTOR, 4801, True)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_given_factorization(cuda_device, monkeypatch, band, cls, batch, shared):
    """A factorization given by the caller, shared or per instance: iterates
    and status of the per-call kernels', a zero pivot reported for its instance."""
    import torch

    b = problems.make_batch(cls, batch, seed=12)
    plan = problems.make_plan(b)
    monkeypatch.setenv("WMPC_STREAM_FRONTIER", "2" if band else "0")
    comp = _compile(monkeypatch, plan, band)
    k = 1 if shared else batch
    args = _dev(b.p_values[:k], b.a_values[:k], b.q, b.l, b.u)
    lx, dinv = comp.factor(args[0], args[1])
    if batch > 1 and not shared:
        dinv[5, 17] = 0.0
    warm = tuple(_dev(*_warm(plan, batch, 4)))
    for w in (None, warm):
        got = comp.engine.solve(*args, warm=w, factor=(lx, dinv))
        assert native.stream_last_launch()["form"] == ("band" if band else "plain")
        status = comp.engine.last_status.clone()
        want = comp.engine.solve(*args, warm=w, factor=(lx, dinv), mode="plain")
        for g, r in zip(got[:3], want[:3]):
            assert torch.equal(g, r)
        zero = (status & native.STATUS_ZERO_PIVOT) != 0
        assert torch.equal(status & ~native.STATUS_ZERO_PIVOT, comp.engine.last_status)
        assert zero.nonzero().flatten().tolist() == ([17] if batch > 1 and not shared else [])


def _sum_qp(n, k, batch, seed):
    """``n`` variables with bounds, one constraint over the first ``k``: a chain of a
    few rows, most subtrees (with k < n) without an entry in it."""
    import scipy.sparse as sp

    from warpmpc_b200.jax_osqp.planning import build_osqp_plan

    rng = np.random.default_rng(seed)
    a = sp.vstack([sp.csr_matrix((np.arange(n) < k).astype(float)[None]), sp.identity(n)]).tocsc()
    bound = np.full(n + 1, 0.5)
    plan = build_osqp_plan(sp.identity(n, format="csc"), a, -bound, bound,
                           OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 600}))
    f = lambda lo, hi, w: rng.uniform(lo, hi, (batch, w)).astype(np.float32)  # noqa: E731
    lim = np.tile(bound.astype(np.float32), (batch, 1))
    return plan, (f(0.5, 2.0, plan.nnz_p), f(0.2, 1.0, plan.nnz_a), f(-2.0, 2.0, n), -lim, lim)


def _short_chain(name, batch):
    if name.startswith("sum"):
        return _sum_qp(60, int(name[3:]), batch, seed=8)
    nu, box, horizon = (2, 1.0, int(name[5:])) if name.startswith("small") else (1, 10.0, int(name[8:]))
    b = problems.make_batch(problems.MPCClass(name, 4, nu, horizon, 5.0, box, 2.0, "small"), batch, seed=3)
    plan = problems.make_plan(b, OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 60}))
    return plan, (b.p_values, b.a_values, b.q, b.l, b.u)


@pytest.mark.parametrize("batch", [40, 9500])
@pytest.mark.parametrize("name", ["small1", "small2", "cartpole1", "cartpole2", "sum60", "sum5"])
def test_band_form_termination_checks_of_short_chains(cuda_device, monkeypatch, name, batch):
    """Fewer chain rows than item warps: warps without a row write their maxima in
    another phase than the rest, and every warp has to come to the same decision."""
    plan, qp = _short_chain(name, batch)
    args = _dev(*qp)
    band, plain = _compile(monkeypatch, plan, 1), _compile(monkeypatch, plan, 0)
    for check in (1, 5):
        for warm in (None, tuple(_dev(*_warm(plan, batch, 8)))):
            got = band.engine.solve(*args, warm=warm, check_termination=check)
            assert native.stream_last_launch()["form"] == "band"
            want = plain.engine.solve(*args, warm=warm, check_termination=check)
            assert native.stream_last_launch()["form"] != "band"
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())
            iters = band.engine.last_iters.cpu().numpy()
            np.testing.assert_array_equal(iters, plain.engine.last_iters.cpu().numpy())
            np.testing.assert_array_equal(band.engine.last_status.cpu().numpy(), plain.engine.last_status.cpu().numpy())
            assert iters.min() < plan.settings.max_iter


@pytest.mark.parametrize("k,batch", [(5, 1), (5, 9500), (60, 33)])
def test_band_form_decoupled_variables(cuda_device, monkeypatch, k, batch):
    """Subtrees that read no chain row: they read the zero row, no sooner than it is written."""
    from oracle.cpu_baseline import CpuOSQP

    plan, qp = _sum_qp(60, k, batch, seed=5)
    comp = _compile(monkeypatch, plan, 1)
    for iters in (1, 2, 7):
        got = comp.engine.solve(*_dev(*qp), max_iter=iters)
        assert native.stream_last_launch()["form"] == "band"
        for g, r in zip(got[:3], CpuOSQP(plan).solve(*qp, max_iter=iters)[:3]):
            np.testing.assert_array_equal(g.cpu().numpy(), r)


def test_given_factorization_in_less_memory(cuda_device, monkeypatch):
    """A given factorization is copied per instance where the memory for it is there;
    else, and in a checked solve, the workspace is the small one and the iterates
    are the same."""
    import torch

    from warpmpc_b200.jax_osqp import solver

    batch = 2500
    b = problems.make_batch(problems.CARTPOLE, batch, seed=12)
    plan = problems.make_plan(b)
    comp = compile_osqp(plan, np.float32, qdldl_backend="cuda", transpose_work=True)
    engine = comp.engine
    args = _dev(b.p_values[:1], b.a_values[:1], b.q, b.l, b.u)
    factor = comp.factor(args[0], args[1])
    least, room = engine.factor_workspace_bytes(batch), 1 << 60
    asked = []

    def allocate(nbytes, device):
        asked.append(nbytes)
        if nbytes > room:
            raise torch.OutOfMemoryError("no room for the copies")
        return torch.empty(int(nbytes), dtype=torch.uint8, device=device), int(nbytes)

    monkeypatch.setattr(solver, "_workspace", allocate)
    want = engine.solve(*args, factor=factor)
    assert len(asked) == 1 and asked[0] > 2 * least
    room = least
    got = [engine.solve(*args, factor=factor)]
    assert asked[1:] == [asked[0], least]
    got.append(engine.solve(*args, factor=factor, workspace=torch.empty(least, dtype=torch.uint8, device=cuda_device)))
    for out in got:
        for g, w in zip(out[:3], want[:3]):
            assert torch.equal(g, w)
    checked = engine.solve(*args, factor=factor, check_termination=5)
    assert asked[3:] == [least] and torch.isfinite(checked[0]).all()
    with pytest.raises(ValueError):
        engine.solve(*args, factor=factor, workspace=torch.empty(least - 1, dtype=torch.uint8, device=cuda_device))
    with pytest.raises(torch.OutOfMemoryError):
        engine.solve(*args)


@pytest.mark.parametrize("check", [0, 5])
def test_band_form_overflowed_instances(cuda_device, monkeypatch, check):
    """Instances whose iterates overflow are reported as in the streaming form, and their
    tiles' other instances are untouched.  (Which of an overflowed instance's values are
    infinite and which are NaN may differ: padding multiplies zeros with its rows.)"""
    batch, broken = 75, [3, 40, 41, 74]
    b = problems.make_batch(problems.CARTPOLE, batch, seed=4)
    plan = problems.make_plan(b, OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 30}))
    p, a, q = b.p_values.copy(), b.a_values.copy(), b.q.copy()
    q[3, 5] = np.inf
    q[40, :] = 3e38
    a[41, 7] = 1e30
    q[74, 0] = np.nan
    band, plain = _compile(monkeypatch, plan, 1), _compile(monkeypatch, plan, 0)
    outs, status = [], []
    for comp in (band, plain):
        outs.append([o.cpu().numpy() for o in comp.engine.solve(*_dev(p, a, q, b.l, b.u), check_termination=check)])
        status.append(comp.engine.last_status.cpu().numpy())
    np.testing.assert_array_equal(*status)
    keep = np.setdiff1d(np.arange(batch), broken)
    for g, w in zip(*outs):
        np.testing.assert_array_equal(g[keep], w[keep])
        # finite in both: the same value
        both = np.isfinite(g) & np.isfinite(w)
        np.testing.assert_array_equal(g[both], w[both])
    assert np.all(status[0][[3, 40, 74]] & native.STATUS_NONFINITE)
