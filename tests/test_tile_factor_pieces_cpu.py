"""The tile factorization's lists as their warps read them: piece by piece.

A list's pieces of 32 words lie in a ring of four, each copied there when the piece
four before it is left.  Copies form one group per tick.  The replay keeps each
piece's copy and checks that the wait at a switch covers it, and that every word
an operation reads belongs to the piece that the ring holds.
"""

import numpy as np
import pytest
import scipy.sparse as sp

from warpmpc_b200 import problems
from warpmpc_b200.jax_osqp import OSQPSettings
from warpmpc_b200.jax_osqp.planning import build_osqp_plan
from warpmpc_b200.schedule import tile_factor_lists

STEP, PIVOT, TICKS, PIECE = 0, 4, 6, 7


def dense_row_plan(n):
    """A diagonal QP with one constraint over all variables: rows of many inputs."""
    a = sp.vstack([sp.csr_matrix(np.ones((1, n))), sp.identity(n)]).tocsc()
    bound = np.ones(n + 1)
    return build_osqp_plan(sp.identity(n, format="csc"), a, -bound, bound, OSQPSettings(**problems.DEFAULT_SETTINGS))


def uncovered_switches(t, first):
    """Switches of one list (from word `first`) to a piece whose copy may still be under way."""
    prog, pos, piece, tick, bad = t["prog"], first, 0, 0, 0
    asked = dict.fromkeys(range(4), -1)  # piece: tick of its copy (-1: before the list starts)
    entered = [0, 0, 0]
    while True:
        x, y = (int(v) for v in prog[pos].view(np.uint32)[:2])
        kind, count = x & 7, x >> 5 & 63
        assert (pos - first) // 32 == piece
        if kind == PIECE and y:
            return bad
        if kind == PIECE:
            ago = tick - entered[2]
            groups = t["piece_wait"][min(ago, t["delay"])]
            # groups complete so far: those of the ticks before this one
            landed = tick if groups < 0 else tick - 1 - groups
            bad += asked[piece + 1] > landed
            asked[piece + 4] = tick
            piece += 1
            entered = [tick] + entered[:2]
            pos = first + 32 * piece
            continue
        if kind == TICKS:
            tick += y
        pos += 1
        if kind not in (PIVOT, TICKS):
            pos += count + (kind == STEP and x >> 4 & 1)
        if x & 8:
            tick += 1


PLANS = [(c.name, lambda c=c: problems.make_plan(problems.make_batch(c, 1, seed=0)))
         for c in (problems.SMALL, problems.CARTPOLE, problems.QUADROTOR)]
PLANS += [(f"dense row {n}", lambda n=n: dense_row_plan(n)) for n in (100, 150, 300, 1000)]


@pytest.mark.parametrize("plan", [p[1] for p in PLANS], ids=[p[0] for p in PLANS])
def test_every_piece_has_landed_when_a_list_goes_on_in_it(plan):
    t = tile_factor_lists(plan().qdldl_plan)
    assert t is not None
    assert [uncovered_switches(t, int(w)) for w in t["warp_off"]] == [0] * t["warps"]
