"""The tile factorization (warpmpc_b200/csrc/tile_factor.cu) on the GPU against the
one-warp-per-tile kernel (``WMPC_DISABLE_TILE_FACTOR=1`` at creation): the same
bits through every stream layout, the same pivot status."""

import numpy as np
import pytest

from warpmpc_b200 import problems
from warpmpc_b200.jax_osqp import OSQPSettings, compile_osqp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env", [{"WMPC_STREAM_BAND": "1"}, {"WMPC_STREAM_BAND": "0", "WMPC_STREAM_FRONTIER": "0"},
                                 {"WMPC_STREAM_FRONTIER": "1"}], ids=["band", "plain", "frontier"])
@pytest.mark.parametrize("cls,batch,adaptive", [(problems.SMALL, 45, False), (problems.CARTPOLE, 9700, True),
                                                (problems.QUADROTOR, 33, True)],
                         ids=lambda v: getattr(v, "name", str(v)))
def test_tile_factor_matches_one_warp(cuda_device, monkeypatch, env, cls, batch, adaptive):
    import torch

    b = problems.make_batch(cls, batch, seed=9)
    settings = {**problems.DEFAULT_SETTINGS, "max_iter": 9}
    if adaptive:
        settings.update(adaptive_rho=True, adaptive_rho_interval=4, adaptive_rho_tolerance=1.5)
    plan = problems.make_plan(b, OSQPSettings(**settings))
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    comps = []
    for off in ("0", "1"):
        monkeypatch.setenv("WMPC_DISABLE_TILE_FACTOR", off)
        comps.append(compile_osqp(plan, np.float32, qdldl_backend="cuda", transpose_work=True, mode="persistent"))
    p = b.p_values.copy()
    p[batch - 3, 1] = np.inf
    args = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (p, b.a_values, b.q, b.l, b.u)]
    outs = [[o.cpu().numpy() for o in c.engine.solve(*args)] for c in comps]
    for g, r in zip(*outs):
        np.testing.assert_array_equal(g, r)
    status = [c.engine.last_status.cpu().numpy() for c in comps]
    np.testing.assert_array_equal(*status)
    assert (status[0] & 4 != 0).nonzero()[0].tolist() == [batch - 3]
    if adaptive:
        assert comps[0].engine.last_rho_updates.sum() > 0


@pytest.mark.parametrize("n", [100, 150, 300, 700])
def test_tile_factor_rows_of_many_inputs(cuda_device, monkeypatch, n):
    """One constraint over all variables: lists that leave several pieces within a
    tick.  L and D^-1 equal the oracle's bit for bit, alone and in the streaming solve."""
    import scipy.sparse as sp
    import torch

    from oracle import osqp_ref, qdldl_ref
    from warpmpc_b200.jax_osqp.planning import build_osqp_plan
    from warpmpc_b200.jax_qdldl import compile_qdldl_variant

    rng = np.random.default_rng(n)
    batch, m = 45, n + 1
    a = sp.vstack([sp.csr_matrix(np.ones((1, n))), sp.identity(n)]).tocsc()
    bound = np.full(m, 0.5)
    plan = build_osqp_plan(sp.identity(n, format="csc"), a, -bound, bound, OSQPSettings(**problems.DEFAULT_SETTINGS))
    p = rng.uniform(0.5, 2.0, (batch, plan.nnz_p)).astype(np.float32)
    av = rng.uniform(0.2, 1.0, (batch, plan.nnz_a)).astype(np.float32)
    kkt = np.ascontiguousarray(osqp_ref.assemble_kkt_values(plan, p, av).T)
    qdldl = compile_qdldl_variant(plan.qdldl_plan, np.float32, backend="cuda", transpose_work=True)
    got = [t.cpu().numpy() for t in qdldl.factor(torch.from_numpy(kkt).cuda())]
    for g, r in zip(got, qdldl_ref.factor(plan.qdldl_plan, kkt)):
        np.testing.assert_array_equal(g, r)
    q = rng.standard_normal((batch, n)).astype(np.float32)
    lim = np.broadcast_to(bound.astype(np.float32), (batch, m))
    monkeypatch.setenv("WMPC_STREAM_BAND", "0")
    comp = compile_osqp(plan, np.float32, qdldl_backend="cuda", transpose_work=True, mode="persistent")
    out = comp.engine.solve(*[torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (p, av, q, -lim, lim)])
    for g, r in zip(out[:3], osqp_ref.solve(plan, p, av, q, -lim, lim)[:3]):
        np.testing.assert_array_equal(g.cpu().numpy(), r)
