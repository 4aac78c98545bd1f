"""What the band form's items wait for, from its host tables.

A subtree's padding slots, and the slots that hold its children's L, read the work
vector's zero row, which item warp 0 writes in the first F phase.  The chain's
sweeps come after that phase, so every subtree has to wait for one chunk at least.
"""

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import osqp_ref
from test_band_cpu import replay
from warpmpc_b200 import native, problems
from warpmpc_b200.jax_osqp import OSQPSettings
from warpmpc_b200.jax_osqp.planning import build_osqp_plan
from warpmpc_b200.schedule import band_tables

USES = 1 << 15


def sum_plan(n, k):
    """``n`` variables with bounds, one constraint over the first ``k``."""
    a = sp.vstack([sp.csr_matrix((np.arange(n) < k).astype(float)[None]), sp.identity(n)]).tocsc()
    bound = np.full(n + 1, 0.5)
    return build_osqp_plan(sp.identity(n, format="csc"), a, -bound, bound, OSQPSettings(**problems.DEFAULT_SETTINGS))


PLANS = {"sum 60": lambda: sum_plan(60, 60), "sum 5 of 60": lambda: sum_plan(60, 5)}
PLANS.update({c.name: lambda c=c: problems.make_plan(problems.make_batch(c, 1, seed=0))
              for c in (problems.SMALL, problems.CARTPOLE, problems.MPCClass("two", 4, 2, 2, 5.0, 1.0, 2.0, "small"))})


@pytest.mark.parametrize("name", list(PLANS))
def test_every_subtree_waits_for_the_chain(name):
    bt = band_tables(PLANS[name]())
    assert bt is not None
    rec = {int(o): bt["rec"][32 * i : 32 * i + 32] for i, o in enumerate(bt["rec_off"])}
    first = [rec[int(w & 0x3FFFFF) * 32] for w in bt["item"].view(np.uint32)[bt["n_pre"] : bt["n_pre"] + bt["nb"]]]
    needs = [int(w[2]) & (USES - 1) for w in first]
    assert min(needs) >= 1 and max(needs) <= bt["n_chunks"]


@pytest.mark.parametrize("k", [60, 5])
def test_band_replay_of_decoupled_variables(k):
    plan = sum_plan(60, k)
    rng = np.random.default_rng(1)

    class Batch:
        batch = 5
        p_values = rng.uniform(0.5, 2.0, (5, plan.nnz_p)).astype(np.float32)
        a_values = rng.uniform(0.2, 1.0, (5, plan.nnz_a)).astype(np.float32)
        q = rng.uniform(-2.0, 2.0, (5, 60)).astype(np.float32)
        u = np.full((5, 61), 0.5, np.float32)
        l = -u

    b = Batch()
    got = replay(plan, band_tables(plan), b, 3)
    ref = osqp_ref.solve(plan, b.p_values, b.a_values, b.q, b.l, b.u, max_iter=3)
    for g, r in zip(got, ref[:3]):
        np.testing.assert_array_equal(g, r)


def unfenced(mb, mf, fence, ahead=4, iters=4):
    """Items of a warp (mb, then mf per iteration) whose iterate is copied back with
    neither the end of a phase nor a fence of its own since it was stored.  Copies run
    ahead as far as their number allows (a full ring only delays them)."""
    per_it, bad = mb + mf, set()
    flying, next_pos, clean = 0, 0, {}  # clean: item: its last store is fenced

    def fill():
        nonlocal flying, next_pos
        while flying < min(ahead, per_it) and next_pos < iters * per_it:
            item = next_pos % per_it
            if not clean.get(item, True):
                bad.add(item)
            flying, next_pos = flying + 1, next_pos + 1

    fill()
    for it in range(iters):
        for item in range(per_it):
            clean[item] = fence
            flying -= 1
            fill()
            if item in (mb - 1, per_it - 1):
                clean = dict.fromkeys(clean, True)
    return bad


@pytest.mark.parametrize("mb", range(9))
def test_items_are_fenced_before_they_are_copied_back(mb):
    for mf in range(9):
        if mb + mf:
            assert not unfenced(mb, mf, bool(native.lib().wmpc_band_item_fence_host(mb, mf))), mf


def test_item_fences_are_left_out_where_phases_are_long():
    assert not native.lib().wmpc_band_item_fence_host(4, 4) and not unfenced(4, 4, False)
    assert unfenced(3, 4, False) and unfenced(4, 3, False) and unfenced(3, 3, False)
