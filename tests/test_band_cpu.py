"""Band form of the persistent solve: its host tables, replayed on the CPU.

One tile runs the kernel's walk in NumPy (chain chunks, B and F items, every
stream and work-vector index bounds-checked, every value an item reads covered
by what it waits for): the iterates equal the oracle's bit for bit.
"""

import numpy as np
import pytest

from oracle import osqp_ref, qdldl_ref
from warpmpc_b200 import problems
from warpmpc_b200.jax_osqp import OSQPSettings
from warpmpc_b200.schedule import band_tables

USES = 1 << 15
F = np.float32


def replay(plan, bt, b, iters, warm=None):
    qp, lanes, B = plan.qdldl_plan, 32, b.batch
    n, npr = qp.n, plan.n
    pick = np.minimum(np.arange(lanes), B - 1)
    kkt = osqp_ref.assemble_kkt_values(plan, b.p_values, b.a_values)[pick]
    lx, _, dinv = qdldl_ref.factor(qp, kkt.T)
    stream = np.full(bt["blen"], np.nan, F)
    state = stream  # the iterates lie in the stream
    lane = np.arange(lanes)

    def at(arr, off, count=lanes, stride=1):
        idx = off + stride * lane
        assert off >= 0 and idx[-1] < arr.size, (off, stride, arr.size)
        return idx

    for e in range(qp.nnz_l):
        stream[at(stream, bt["lpos"][e], stride=4)] = lx[e]
        stream[at(stream, bt["lpos2"][e], stride=4)] = lx[e]
    for k in range(n):
        stream[at(stream, bt["dpos"][k])] = dinv[k]
    for p in bt["pad"]:
        stream[at(stream, p, stride=4)] = 0.0
    w = (np.zeros((B, npr), F), np.zeros((B, plan.m), F), np.zeros((B, plan.m), F)) if warm is None else warm
    cs = lambda a: np.asarray(a, F)  # noqa: E731
    x0, z0, y0 = w[0] * cs(plan.scaling_dinv), w[1] * cs(plan.scaling_e), w[2] * cs(plan.y_scale)
    qs, ls, us = b.q * cs(plan.q_scale), b.l * cs(plan.scaling_e), b.u * cs(plan.scaling_e)
    for k in range(n):
        io, po = bt["iter_off"][k], bt["param_off"][k]
        if k < npr:
            state[at(state, io)] = x0[pick, k]
            stream[at(stream, po)] = qs[pick, k]
        else:
            r = k - npr
            for j, v in enumerate((z0, y0)):
                state[at(state, io + j, stride=2)] = v[pick, r]
            for j, v in enumerate((ls, us)):
                stream[at(stream, po + j, stride=2)] = v[pick, r]
    sigma, alpha = F(plan.settings.sigma), F(plan.settings.alpha)
    oma = F(1.0) - alpha
    fl = lambda i: np.array([i], np.int32).view(F)[0]  # noqa: E731
    T, T4, U, n_pre, n_yr = bt["T"], bt["T4"], bt["units"], bt["n_pre"], bt["n_yr"]
    vzero = T4 + 4 * U
    V = np.full((vzero + 1 + n_pre, lanes), np.nan, F)
    YR = np.full((n_yr + 1, lanes), np.nan, F)
    V[T : vzero + 1] = 0.0
    YR[n_yr] = 0.0

    def rec(kind, soff, poff):
        if kind & 1:
            return (state[at(state, soff, stride=2)], state[at(state, soff + 1, stride=2)],
                    stream[at(stream, poff, stride=2)], stream[at(stream, poff + 1, stride=2)])
        return (state[at(state, soff)], stream[at(stream, poff)])

    def rhs_of(kind, rinv, r):
        return r[0] - rinv * r[1] if kind & 1 else sigma * r[0] - r[1]

    def update(kind, xs, rho, rinv, soff, r):
        if kind & 1:
            z, y, lo, hi = r
            rz = z - rinv * y
            zr = alpha * (rz + rinv * xs) + oma * z
            zn = zr + rinv * y
            zn = np.where(zn < lo, lo, zn)
            zn = np.where(zn > hi, hi, zn)
            yn = y + rho * (zr - zn)
            state[at(state, soff, stride=2)] = zn
            state[at(state, soff + 1, stride=2)] = yn
            return zn - rinv * yn
        xn = alpha * xs + oma * r[0]
        state[at(state, soff)] = xn
        return sigma * xn - r[1]

    def units(base, count):  # the L entries of consecutive units
        return [stream[at(stream, base + 128 * (e >> 2) + (e & 3), stride=4)] for e in range(4 * count)]

    def width(kind):
        return 64 if kind & 1 else 32

    # records and item offsets travel in the stream
    for row, at_ in zip(bt["rec"].reshape(-1, 32), bt["rec_off"]):
        assert np.all(np.isnan(stream[at_ : at_ + 32])) and at_ % 32 == 0
        stream[at_ : at_ + 32] = row.view(F)
    n_b, items = n_pre + bt["nb"], []
    for word in bt["item"].view(np.uint32).astype(int):
        at_, size = (word & 0x3FFFFF) * 32, (word >> 22) * 32
        assert 0 < size * 4 <= bt["item_bytes"] and at_ + size <= bt["blen"]
        rows = int(stream[at_ : at_ + 1].view(np.int32)[0]) >> 27 & 31
        items.append((at_ + 32 * rows, stream[at_ : at_ + 32 * rows].view(np.int32), at_ + size))
    assert len(items) == n_b + n_pre + T

    def b_phase(it):
        for i in range(n_b):
            off, w, end = items[i]
            z, yr, need, uses = int(w[0]), int(w[1]) // 128, int(w[2]) & (USES - 1), bool(w[2] & USES) or i < n_pre
            nu, nc, kr = z & 15, z >> 4 & 15, z >> 8 & 15
            rows = [int(v) // 128 for v in w[16 : 16 + 4 * nu]]
            assert len(rows) == 4 * nu and nc <= 2 and yr < n_yr and need <= bt["n_chunks"]
            for t in rows:
                assert 0 <= t < V.shape[0]
                assert bt["n_chunks"] - t // bt["chunk_cols"] <= need if t < T else t == vzero or (uses and t > vzero)
            L = units(off, nu)
            q = off + 128 * nu
            xr = None
            if it > 0:
                corr = np.zeros(lanes, F)
                for t, l in zip(rows, L):
                    corr = corr + l * V[t]
                xr = YR[yr] * stream[at(stream, q)] - corr
            if i < n_pre:
                vo = int(w[3]) // 128
                assert vzero < vo < V.shape[0] and q + 32 == end
                if it > 0:
                    V[vo] = xr
                continue
            assert w[3] == q
            acc = None
            for c in range(nc + 1):  # the root, then its children
                kc, rho, rinv = z >> (8 + 4 * c) & 15, fl(w[4 + 4 * c]), fl(w[5 + 4 * c])
                soff = q + 32 + width(kc)
                r = rec(kc, soff, q + 32)
                l = None if c == 0 else L[4 * nu - c]
                v = rhs_of(kc, rinv, r)
                if it > 0:
                    xs = xr if c == 0 else v * stream[at(stream, q)] - (F(0) + l * xr)
                    v = update(kc, xs, rho, rinv, soff, r)
                acc = v if c == 0 else acc - l * v
                q = soff + width(kc)
            assert q == end
            YR[yr] = acc

    def f_phase(it):
        for i in range(n_pre + T):
            off, w, end = items[n_b + i]
            z, vo, out = int(w[0]), int(w[1]) // 128, int(w[2])
            nu, kind, uses = z & 255, z >> 8 & 15, z & USES
            assert vo == (i - n_pre if i >= n_pre else vzero + 1 + i) and (out < 0) == (i >= n_pre)
            rows = [int(v) // 128 for v in w[8 : 8 + 4 * nu]]
            assert len(rows) == 4 * nu and off + 128 * nu + 2 * width(kind) == end and w[3] == off + 128 * nu
            soff = off + 128 * nu + width(kind)
            r = rec(kind, soff, off + 128 * nu)
            acc = update(kind, V[vo].copy(), fl(w[4]), fl(w[5]), soff, r) if it > 0 else rhs_of(kind, fl(w[5]), r)
            if it < iters:
                for t, l in zip(rows, units(off, nu)):
                    assert 0 <= t <= n_yr and (uses or i < n_pre or not n_yr - n_pre <= t < n_yr)
                    acc = acc - l * YR[t]
                if out >= 0:
                    YR[out // 128] = acc
                else:
                    V[vo] = acc

    def columns():
        for ch in range(bt["n_chunks"]):
            off, ub, cols, rows = map(int, bt["chunk"][4 * ch : 4 * ch + 4])
            cols, nf = cols & 255, cols >> 8
            far = bt["far"].reshape(-1, 4)[bt["far_ptr"][ch] : bt["far_ptr"][ch] + nf]
            assert cols % 4 == 0 and cols <= bt["chunk_cols"] and ub + 128 * cols <= bt["chunk_bytes"]
            for j in range(cols):
                t = ch * bt["chunk_cols"] + j
                word = int(bt["col_word"][t])
                u, u0 = U - 1 + (word & 1), word >> 1
                assert (u0 + u) * 512 <= ub and rows >= min(T, t + 4 * U + 1)
                fr = [(int(f[1]) // 128, stream[at(stream, off + int(f[2]) // 4, stride=4)]) for f in far if f[0] == j]
                assert all(t + 4 * U < r < rows for r, _ in fr) and all(int(f[2]) < ub for f in far)
                yield t, units(off + 128 * u0, u), fr, stream[at(stream, off + ub // 4 + 32 * j)]

    b_phase(0)
    f_phase(0)
    for it in range(1, iters + 1):
        cols = list(columns())
        assert [c[0] for c in cols] == list(range(T4))
        for t, win, far, _ in cols:
            for j, l in enumerate(win):
                V[t + 1 + j] = V[t + 1 + j] - l * V[t]
            for r, l in far:
                V[r] = V[r] - l * V[t]
        for t, win, far, d in reversed(cols):
            corr = np.zeros(lanes, F)
            for j, l in enumerate(win):
                corr = corr + l * V[t + 1 + j]
            for r, l in far:
                corr = corr + l * V[r]
            V[t] = V[t] * d - corr
        b_phase(it)
        f_phase(it)
    x, z, y = np.empty((B, npr), F), np.empty((B, plan.m), F), np.empty((B, plan.m), F)
    for k in range(n):
        io = bt["iter_off"][k]
        if k < npr:
            x[:, k] = state[at(state, io)][:B]
        else:
            z[:, k - npr] = state[at(state, io, stride=2)][:B]
            y[:, k - npr] = state[at(state, io + 1, stride=2)][:B]
    return x * cs(plan.scaling_d), z * cs(plan.scaling_einv), y * cs(plan.y_unscale)


CLASSES = [problems.SMALL, problems.MPCClass("c20", 4, 1, 20, 5.0, 10.0, 2.0, "small"),
           problems.MPCClass("q5", 12, 4, 5, 10.0, 2.0, 1.0, "quadrotor"),
           problems.MPCClass("one", 3, 2, 1, 5.0, 1.0, 2.0, "small"),
           problems.MPCClass("wide", 5, 7, 4, 5.0, 1.0, 2.0, "small")]


@pytest.mark.parametrize("cls", CLASSES, ids=[c.name for c in CLASSES])
def test_band_replay_bitexact(cls):
    b = problems.make_batch(cls, 7, seed=3)
    plan = problems.make_plan(b)
    bt = band_tables(plan)
    if bt is None:
        pytest.skip("no band form")
    got = replay(plan, bt, b, 3)
    ref = osqp_ref.solve(plan, b.p_values, b.a_values, b.q, b.l, b.u, max_iter=3)
    for g, r in zip(got, ref[:3]):
        np.testing.assert_array_equal(g, r)
    warm = ref[:3]
    got = replay(plan, bt, b, 2, warm)
    ref = osqp_ref.solve_warm_start(plan, b.p_values, b.a_values, b.q, b.l, b.u, *warm, max_iter=2)
    for g, r in zip(got, ref[:3]):
        np.testing.assert_array_equal(g, r)


@pytest.mark.parametrize("perm", ["natural", "random"])
def test_band_tables_other_orderings(perm):
    """Orderings whose factor is no band: either no band form, or one whose replay is exact."""
    b = problems.make_batch(problems.MPCClass("s3", 4, 2, 3, 5.0, 1.0, 2.0, "small"), 5, seed=1)
    nk = b.p_matrix0.shape[0] + b.a_matrix0.shape[0]
    p = np.arange(nk) if perm == "natural" else np.random.default_rng(0).permutation(nk)
    plan = problems.make_plan(b, OSQPSettings(**problems.DEFAULT_SETTINGS), perm=p)
    bt = band_tables(plan)
    if bt is not None:
        got = replay(plan, bt, b, 2)
        ref = osqp_ref.solve(plan, b.p_values, b.a_values, b.q, b.l, b.u, max_iter=2)
        for g, r in zip(got, ref[:3]):
            np.testing.assert_array_equal(g, r)


def test_band_form_of_the_benchmark_patterns():
    """The benchmark classes have the form, with the window they were measured in."""
    for cls, units in ((problems.SMALL, 2), (problems.CARTPOLE, 2), (problems.QUADROTOR, 4)):
        bt = band_tables(problems.make_plan(problems.make_batch(cls, 1, seed=0)))
        assert bt is not None and bt["units"] == units
