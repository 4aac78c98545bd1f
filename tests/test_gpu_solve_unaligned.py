"""The streamed per-call solve where the tensor copies' 16-byte rule does not
hold (odd batches, arrays that start 4 bytes off): the one-lane kernel's bits."""

import numpy as np
import pytest

from oracle import qdldl_ref
from warpmpc_b200 import problems
from warpmpc_b200.jax_qdldl import compile_qdldl_variant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,horizon", [(4, 2), (4, 8), (4, 20)])
@pytest.mark.parametrize("batch", [9501, 30001, 60001])
def test_unaligned_solve_of_short_patterns(cuda_device, monkeypatch, nx, horizon, batch):
    """Several tiles per SM: few stages and many CTAs, or the one-lane kernel."""
    import torch

    b = problems.make_batch(problems.MPCClass("x", nx, 1, horizon, 5.0, 10.0, 2.0, "small"), 2, seed=8)
    qp = problems.make_plan(b).qdldl_plan
    comp = compile_qdldl_variant(qp, np.float32, backend="cuda", transpose_work=True)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    lx, dinv, rhs = (torch.randn(k, batch, generator=gen, device="cuda") for k in (qp.nnz_l, qp.n, qp.n))
    got = comp.solve(0.02 * lx, dinv, rhs).clone()
    monkeypatch.setenv("WMPC_SOLVE_STREAM_OFF", "1")
    assert torch.equal(got, comp.solve(0.02 * lx, dinv, rhs))


@pytest.mark.parametrize("batch,shift", [(1, 0), (31, 0), (33, 1), (64, 1), (4803, 0)])
def test_unaligned_solve_matches_one_lane(cuda_device, monkeypatch, batch, shift):
    import torch

    b = problems.make_batch(problems.CARTPOLE, 2, seed=8)
    qp = problems.make_plan(b).qdldl_plan
    comp = compile_qdldl_variant(qp, np.float32, backend="cuda", transpose_work=True)
    gen = torch.Generator(device="cuda").manual_seed(batch)

    def draw(rows):  # [rows, batch], `shift` floats into its allocation
        v = torch.randn(rows * batch + shift, generator=gen, device="cuda")
        return v[shift:].view(rows, batch)

    lx, dinv, rhs = 0.02 * draw(qp.nnz_l), draw(qp.n), draw(qp.n)
    got = comp.solve(lx, dinv, rhs).clone()
    monkeypatch.setenv("WMPC_SOLVE_STREAM_OFF", "1")
    want = comp.solve(lx, dinv, rhs)
    assert torch.equal(got, want)
    sl = slice(max(0, batch - 40), batch)
    ref = qdldl_ref.solve(qp, *(t.cpu().numpy()[:, sl] for t in (lx, dinv, rhs)))
    np.testing.assert_array_equal(got.cpu().numpy()[:, sl], ref)
