"""The tile factorization's lists, replayed on the CPU.

The warps' lists run tick by tick in NumPy: a slot is read only where an earlier
tick or the same warp has written it, rewritten only where no other warp reads
it in the same tick, and a load is used only `delay` ticks later.  L, D and D^-1
equal the oracle's bit for bit.
"""

import numpy as np
import pytest

from oracle import osqp_ref, qdldl_ref
from warpmpc_b200 import problems
from warpmpc_b200.schedule import tile_factor_lists

F = np.float32
STEP, INPUTS, ZEROS, CONSTS, PIVOT, LOAD, TICKS, PIECE = range(8)


def replay(qp, t, values):
    """values: [nnz_kkt, lanes]"""
    lanes = values.shape[1]
    lx, dinv = np.full((qp.nnz_l, lanes), np.nan, F), np.full((qp.n, lanes), np.nan, F)
    v = np.full((t["slots"], lanes), np.nan, F)
    wrote = [(-1, -1)] * t["slots"]  # tick, warp
    read = [{} for _ in range(t["slots"])]  # warp: tick
    loading = {}
    prog, pos = t["prog"], list(t["warp_off"])
    wait = [0] * t["warps"]  # ticks the warp still sits out
    ended = [False] * t["warps"]
    fl = lambda w: np.int32(w).view(F)  # noqa: E731

    def get(s, tick, w):
        assert 0 < s < t["slots"] and (wrote[s][0] < tick or wrote[s][1] == w) and s not in loading, (s, tick, w)
        read[s][w] = tick
        return v[s]

    def put(s, x, tick, w):
        assert 0 < s < t["slots"]
        assert all(k != tick or q == w for q, k in read[s].items()) and (wrote[s][0] < tick or wrote[s][1] == w)
        v[s] = x
        wrote[s] = (tick, w)

    low = lambda x: int(x) >> 7 & 2047  # noqa: E731
    high = lambda x: int(x) >> 18 & 2047  # noqa: E731
    for tick in range(t["ticks"] + 1):
        for w in range(t["warps"]):
            if wait[w]:
                wait[w] -= 1
                continue
            alone = True
            while not ended[w]:
                h = [int(x) for x in prog[pos[w]].view(np.uint32)]
                kind, cnt = h[0] & 7, h[0] >> 5 & 63
                body = pos[w] + 1 + (kind == STEP and h[0] >> 4 & 1)
                if kind not in (TICKS, PIECE):
                    # one piece (the lists start at a multiple of 32 words from one another)
                    first = pos[w] - t["warp_off"][w]
                    end = body + (cnt if kind not in (PIVOT, TICKS) else 0) - t["warp_off"][w]
                    assert first // 32 == (end - 1) // 32
                words = prog[body : body + cnt]
                start, pos[w] = pos[w], body + (cnt if kind not in (PIVOT, TICKS, PIECE) else 0)
                if kind == STEP:
                    ds, c = h[0] >> 21, high(h[1])
                    val = get(low(h[1]), tick, w).copy()
                    dcol = get(c, tick, w).copy()
                    lval = val * dcol
                    dk = get(ds, tick, w) - val * lval
                    assert np.all(np.isnan(lx[h[2]])) and h[3] == h[2]
                    lx[h[2]] = lval
                    put(ds, dk, tick, w)
                    if h[0] & 16:
                        row = int(prog[start + 1, 0])
                        dinv[row] = F(1) / dk
                        put(ds, dinv[row], tick, w)
                    ups = [u for u in words.reshape(-1) if u]
                    assert len({low(u) for u in ups}) == len(ups)
                    for u in ups:
                        put(low(u), get(low(u), tick, w) - (get(high(u), tick, w) * dcol) * val, tick, w)
                elif kind == INPUTS:
                    for x in words:
                        s = low(x[0])
                        since, by = loading.pop(s)
                        assert by == w and tick - since >= t["delay"]
                        put(s, v[s] * fl(x[1]) + fl(x[2]), tick, w)
                elif kind == ZEROS:
                    for x in words.reshape(-1):
                        if x:
                            put(low(x), F(0), tick, w)
                elif kind == CONSTS:
                    for x in words.reshape(-1, 2):
                        if x[0]:
                            put(low(x[0]), fl(x[1]), tick, w)
                elif kind == PIVOT:
                    dinv[h[2]] = F(1) / get(low(h[1]), tick, w)
                    put(low(h[1]), dinv[h[2]], tick, w)
                elif kind == LOAD:
                    assert h[1] == 0
                    for x in words.reshape(-1):
                        if x:
                            s = int(x) >> 20
                            assert s not in loading
                            put(s, values[int(x) & 0xFFFFF], tick, w)
                            loading[s] = (tick, w)
                elif kind == TICKS:
                    assert alone and h[1] > 0  # nothing else in these ticks
                    wait[w] = h[1] - 1
                    break
                elif h[1]:
                    assert tick == t["ticks"]
                    ended[w] = True
                else:
                    pos[w] = t["warp_off"][w] + ((start - t["warp_off"][w]) // 32 + 1) * 32
                    continue
                alone = False
                if h[0] & 8:
                    break
    assert all(ended)
    return lx, dinv


CLASSES = [problems.SMALL, problems.CARTPOLE, problems.MPCClass("q5", 12, 4, 5, 10.0, 2.0, 1.0, "quadrotor"),
           problems.MPCClass("one", 4, 2, 1, 5.0, 1.0, 2.0, "small"), problems.QUADROTOR]


@pytest.mark.parametrize("cls", CLASSES, ids=lambda c: c.name)
def test_tile_factor_replay_bitexact(cls):
    b = problems.make_batch(cls, 3, seed=2)
    plan = problems.make_plan(b)
    qp = plan.qdldl_plan
    t = tile_factor_lists(qp)
    assert t is not None and t["slots"] * 128 + t["warps"] * 2048 + 128 <= 227 * 1024
    kkt = osqp_ref.assemble_kkt_values(plan, b.p_values, b.a_values).T
    lx, dinv = replay(qp, t, kkt)
    ref_lx, _, ref_dinv = qdldl_ref.factor(qp, kkt)
    np.testing.assert_array_equal(dinv, ref_dinv)
    np.testing.assert_array_equal(lx, ref_lx)
