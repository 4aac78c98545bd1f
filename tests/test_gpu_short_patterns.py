"""Patterns of a few chunks in every schedule form: the streaming kernels' rings hold
more chunks than such a pattern has, so a chunk's records are asked for while an
iteration before is still being released.  Iterates equal the oracle's bit for bit.
"""

import numpy as np
import pytest
import scipy.sparse as sp

from oracle.cpu_baseline import CpuOSQP
from warpmpc_b200 import native, problems
from warpmpc_b200.jax_osqp import OSQPSettings, compile_osqp, solve_classes
from warpmpc_b200.jax_osqp.planning import build_osqp_plan

pytestmark = pytest.mark.gpu

FORMS = {"plain": {"WMPC_STREAM_BAND": "0", "WMPC_STREAM_FRONTIER": "0"},
         "frontier": {"WMPC_STREAM_BAND": "0", "WMPC_STREAM_FRONTIER": "1"},
         "band": {"WMPC_STREAM_BAND": "1"}, "default": {}}
SETTINGS = OSQPSettings(**{**problems.DEFAULT_SETTINGS, "max_iter": 20})


def _pattern(name, batch):
    if name == "box":  # decoupled variables with bounds: no chain, hence no band form
        plan = build_osqp_plan(sp.identity(9, format="csc"), sp.identity(9, format="csc"), -np.ones(9), np.ones(9),
                               SETTINGS)
        rng = np.random.default_rng(3)
        f = lambda lo, hi, w: rng.uniform(lo, hi, (batch, w)).astype(np.float32)  # noqa: E731
        return plan, (f(0.5, 2.0, 9), f(0.5, 2.0, 9), f(-3.0, 3.0, 9), f(-2.0, -1.0, 9), f(1.0, 2.0, 9))
    nu, box = (2, 1.0) if name.startswith("small") else (1, 10.0)
    cls = problems.MPCClass(name, 4, nu, int(name[-1]), 5.0, box, 2.0, "small")
    b = problems.make_batch(cls, batch, seed=3)
    return problems.make_plan(b, SETTINGS), (b.p_values, b.a_values, b.q, b.l, b.u)


def _engine(monkeypatch, plan, form):
    with monkeypatch.context() as m:
        for k, v in FORMS[form].items():
            m.setenv(k, v)
        return compile_osqp(plan, np.float32, qdldl_backend="cuda", transpose_work=True, mode="persistent").engine


def _dev(arrays):
    import torch

    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("name", ["box", "small1", "small2", "small3", "cartpole1", "cartpole3"])
def test_short_patterns_bitexact(cuda_device, monkeypatch, name, form):
    for batch in (40, 9500):
        plan, qp = _pattern(name, batch)
        engine = _engine(monkeypatch, plan, form)
        for warm in (None, [0.1 * np.random.default_rng(1).standard_normal((batch, k)).astype(np.float32)
                            for k in (plan.n, plan.m, plan.m)]):
            got = engine.solve(*_dev(qp), warm=None if warm is None else tuple(_dev(warm)))
            launch = native.stream_last_launch()["form"]
            assert form == "default" or launch == ("plain" if name == "box" and form == "band" else form)
            for g, r in zip(got[:3], CpuOSQP(plan).solve(*qp, warm=warm)[:3]):
                np.testing.assert_array_equal(g.cpu().numpy(), r)


def test_short_and_long_patterns_in_one_launch(cuda_device, monkeypatch):
    """Classes of few and of many chunks share a launch and its rings."""
    work, ref = [], []
    for name in ("cartpole9", "small1", "small3"):
        plan, qp = _pattern(name, 500)
        work.append((_engine(monkeypatch, plan, "plain"), *_dev(qp), None))
        ref.append(CpuOSQP(plan).solve(*qp))
    for out, r in zip(solve_classes(work), ref):
        for g, w in zip(out[:3], r[:3]):
            np.testing.assert_array_equal(g.cpu().numpy(), w)
    assert native.stream_last_launch()["form"] == "plain"
