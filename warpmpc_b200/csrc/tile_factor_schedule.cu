// Host scheduler of the tile factorization (see tile_factor.cuh): list scheduling
// of the row programs' steps by their longest path to the end.
#include <algorithm>
#include <climits>
#include <cstring>
#include <queue>

#include "tile_factor.cuh"

namespace wmpc {

namespace {

int bits(float v) {
  int b;
  std::memcpy(&b, &v, 4);
  return b;
}

float real(int b) {
  float v;
  std::memcpy(&v, &b, 4);
  return v;
}

}  // namespace

size_t tile_factor_smem(int slots) { return (size_t)slots * 128 + kTfWarps * 2048 + 128; }

void place_tile_factor(const int* boff, const int* foff, const int* doff, HostTileFactor* t) {
  for (size_t e = 0; e < t->step_at.size(); ++e) {
    t->prog[t->step_at[e]] = boff[e];
    t->prog[t->step_at[e] + 1] = foff[e];
  }
  for (size_t k = 0; k < t->row_at.size(); ++k) t->prog[t->row_at[k]] = doff[k];
}

bool schedule_tile_factor(const HostPattern& hp, const std::vector<int>& init_slot, HostTileSchedule* out,
                          std::string* why) {
  const int n = hp.n, S = hp.nnz_l, N = S + n;  // tasks: steps, then the rows' inits
  std::vector<int> step_of_l(std::max(S, 1), -1);
  for (int k = 0; k < n; ++k)
    for (int e = hp.proc_ptr[k]; e < hp.proc_ptr[k + 1]; ++e) {
      step_of_l[hp.proc_lidx[e]] = e;
    }
  auto end_of = [&](int k) { return hp.proc_ptr[k + 1] > hp.proc_ptr[k] ? hp.proc_ptr[k + 1] - 1 : S + k; };
  auto first_of = [&](int k) { return hp.proc_ptr[k + 1] > hp.proc_ptr[k] ? hp.proc_ptr[k] : -1; };
  // ---- dependences ----
  std::vector<std::vector<int>> succ(N);
  std::vector<int> npred(N, 0), cost(N);
  auto dep = [&](int a, int b) {
    succ[a].push_back(b);
    ++npred[b];
  };
  out->upd.assign(S, {});
  auto& upd = out->upd;
  std::vector<int> final_by(S);  // the task after which a step's y is final
  for (int k = 0; k < n; ++k) {
    const int p0 = hp.proc_ptr[k], p1 = hp.proc_ptr[k + 1], ni = 1 + hp.init_ptr[k + 1] - hp.init_ptr[k];
    for (int e = p0; e < p1; ++e) final_by[e] = S + k;
    cost[S + k] = 40 + 8 * (ni + p1 - p0);
    std::vector<char> seen(p1 - p0, 0);
    for (int i = hp.init_ptr[k]; i < hp.init_ptr[k + 1]; ++i) {
      const int s = init_slot[i];
      if (s < 0 || s >= p1 - p0 || seen[s]) {
        *why = "a row has two inputs for one entry";
        return false;
      }
      seen[s] = 1;
    }
    std::vector<std::pair<int, int>> local;  // {column, step index}
    for (int e = p0; e < p1; ++e) local.push_back({hp.proc_cols[e], e - p0});
    std::sort(local.begin(), local.end());
    if (first_of(k) >= 0) dep(S + k, p0);
    for (int e = p0; e < p1; ++e) {
      const int c = hp.proc_cols[e], nu = hp.proc_offsets[e];
      cost[e] = 110 + 9 * nu + (e + 1 == p1 ? 60 : 0);
      if (nu > 112) {
        *why = "a column is too long";
        return false;
      }
      if (e + 1 < p1) dep(e, e + 1);
      dep(end_of(c), e);
      for (int q = 0; q < nu; ++q) {
        const int l = hp.lp[c] + q, j = hp.li[l], src = step_of_l[l];
        const auto it = std::lower_bound(local.begin(), local.end(), std::make_pair(j, INT_MIN));
        if (src < 0 || j >= k || it == local.end() || it->first != j || it->second <= e - p0) {
          *why = "a row program is out of order";
          return false;
        }
        upd[e].push_back({it->second, src});
        dep(final_by[src], e);
        final_by[p0 + it->second] = e;
      }
    }
  }
  // ---- longest path to the end ----
  std::vector<int> tail(N, 0);
  int total = 0;
  auto settle = [&](int t) {
    int m = 0;
    for (int s : succ[t]) m = std::max(m, tail[s]);
    tail[t] = m + cost[t];
    total = std::max(total, tail[t]);
  };
  for (int k = n - 1; k >= 0; --k) {
    for (int e = hp.proc_ptr[k + 1] - 1; e >= hp.proc_ptr[k]; --e) settle(e);
    settle(S + k);
  }
  auto late = [&](int t) { return total - tail[t]; };  // latest start, were there warps enough
  std::vector<int> rows(n), by_late(N);
  for (int k = 0; k < n; ++k) rows[k] = k;
  std::stable_sort(rows.begin(), rows.end(), [&](int a, int b) { return late(S + a) < late(S + b); });
  for (int t = 0; t < N; ++t) by_late[t] = t;
  std::stable_sort(by_late.begin(), by_late.end(), [&](int a, int b) { return late(a) < late(b); });
  // ---- schedule ----
  const int W = kTfWarps;
  auto schedule = [&](int look, std::vector<int> npred, HostTileSchedule* result) -> bool {
    HostTileSchedule& H = *result;
    std::vector<int> tick(N, -1), warp(N, -1), load_tick(n, -1), dep_tick(N, -1), dep_warp(N, -1);
    auto& ops = H.ops;
    ops.assign(W, {});
    struct Ready {
      int tail, task, warp;  // warp -1: any
      bool operator<(const Ready& o) const { return tail != o.tail ? tail < o.tail : task > o.task; }
    };
    std::vector<Ready> next;                      // ready from the next tick on
    std::vector<std::vector<Ready>> later(kTfDelay + 1);  // inits, by tick modulo
    int done = 0, at_row = 0, at_late = 0, t = 0;
    for (; done < N; ++t) {
      if (t > 64 * N) {
        *why = "the factorization's schedule does not end";
        return false;
      }
      std::priority_queue<Ready> ready(std::less<Ready>(), std::move(next));
      next.clear();
      for (const Ready& r : later[t % (kTfDelay + 1)]) ready.push(r);
      later[t % (kTfDelay + 1)].clear();
      std::vector<int> load(W, 0);
      while (!ready.empty()) {
        const Ready r = ready.top();
        ready.pop();
        int w = r.warp;
        if (w < 0) w = static_cast<int>(std::min_element(load.begin(), load.end()) - load.begin());
        if (load[w] > 0 && load[w] + cost[r.task] > kTfTick) {
          next.push_back({r.tail, r.task, r.task >= S ? r.warp : -1});
          continue;
        }
        load[w] += cost[r.task];
        tick[r.task] = t;
        warp[r.task] = w;
        ops[w].push_back({t, r.task});
        ++done;
        for (int s : succ[r.task]) {
          if (dep_tick[s] == t && dep_warp[s] != w) dep_warp[s] = -2;
          else dep_warp[s] = w;
          dep_tick[s] = t;
          if (--npred[s] > 0) continue;
          if (dep_warp[s] >= 0) ready.push({tail[s], s, w});  // the same warp may go on at once
          else next.push_back({tail[s], s, -1});
        }
      }
      while (at_late < N && tick[by_late[at_late]] >= 0) ++at_late;
      const int front = at_late < N ? late(by_late[at_late]) : total;
      for (; at_row < n && late(S + rows[at_row]) <= front + look; ++at_row) {
        const int k = rows[at_row], ni = 1 + hp.init_ptr[k + 1] - hp.init_ptr[k];
        const int w = static_cast<int>(std::min_element(load.begin(), load.end()) - load.begin());
        if (load[w] > kTfTick) break;
        load[w] += 20 + 12 * ni;
        load_tick[k] = t;
        ops[w].push_back({t, N + k});
        later[(t + kTfDelay) % (kTfDelay + 1)].push_back({tail[S + k], S + k, w});
      }
    }
    H.ticks = t;
    // ---- slots ----
    struct Value {
      int from, to, id;  // id: step e: its row's slot, S + k: d of row k
    };
    std::vector<Value> values;
    std::vector<int> last_y(tick.begin(), tick.begin() + S), last_d(n);
    for (int k = 0; k < n; ++k) last_d[k] = tick[end_of(k)];
    for (int e = 0; e < S; ++e) {
      last_d[hp.proc_cols[e]] = std::max(last_d[hp.proc_cols[e]], tick[e]);
      for (const auto& u : upd[e]) last_y[u.second] = std::max(last_y[u.second], tick[e]);
    }
    for (int k = 0; k < n; ++k) {
      std::vector<char> has(hp.proc_ptr[k + 1] - hp.proc_ptr[k], 0);
      for (int i = hp.init_ptr[k]; i < hp.init_ptr[k + 1]; ++i) has[init_slot[i]] = 1;
      for (int e = hp.proc_ptr[k]; e < hp.proc_ptr[k + 1]; ++e)
        values.push_back({has[e - hp.proc_ptr[k]] ? load_tick[k] : tick[S + k], last_y[e], e});
      values.push_back({load_tick[k], last_d[k], S + k});
    }
    std::stable_sort(values.begin(), values.end(), [](const Value& a, const Value& b) { return a.from < b.from; });
    std::vector<int> spare;
    auto& slot = H.slot;
    slot.assign(S + n, 0);
    std::priority_queue<std::pair<int, int>, std::vector<std::pair<int, int>>, std::greater<std::pair<int, int>>> busy;
    H.slots = 1;
    for (const Value& v : values) {
      while (!busy.empty() && busy.top().first < v.from) {
        spare.push_back(busy.top().second);
        busy.pop();
      }
      int s;
      if (spare.empty()) {
        s = H.slots++;
      } else {
        s = spare.back();
        spare.pop_back();
      }
      slot[v.id] = s;
      busy.push({v.to, s});
    }
    return true;
  };
  // Rows that start early keep every warp busy and take slots: as early as the
  // slots of two CTAs per SM allow, else of one.
  HostTileSchedule best, one;
  best.slots = INT_MAX;
  for (int ticks : {kTfDelay + 8, kTfDelay + 2, kTfDelay}) {
    if (!schedule(kTfTick * ticks, npred, &one)) return false;
    if (one.slots <= kTfSlots2 || (best.slots > kTfSlots && one.slots < best.slots)) std::swap(best, one);
    if (best.slots <= kTfSlots2) break;
  }
  if (best.slots > kTfSlots) {
    *why = "the factorization's values in flight do not fit (" + std::to_string(best.slots) + " slots)";
    return false;
  }
  out->ops.swap(best.ops);
  out->slot.swap(best.slot);
  out->slots = best.slots;
  out->ticks = best.ticks;
  return true;
}

bool emit_tile_factor(const HostTileSchedule& sched, const HostPattern& hp, const std::vector<int>& init_slot,
                      const int* kin, int np, int na, HostTileFactor* out, std::string* why) {
  HostTileFactor& H = *out;
  H = HostTileFactor{};
  H.slots = sched.slots;
  H.ticks = sched.ticks;
  const int n = hp.n, S = hp.nnz_l, N = S + n, W = kTfWarps;
  const auto &ops = sched.ops;
  const auto &slot = sched.slot;
  const auto &upd = sched.upd;
  std::vector<int> row_of(S);
  for (int k = 0; k < n; ++k)
    for (int e = hp.proc_ptr[k]; e < hp.proc_ptr[k + 1]; ++e) row_of[e] = k;
  // ---- the lists ----
  H.step_at.assign(S, 0);
  H.row_at.assign(n, 0);
  for (int w = 0; w < W; ++w) {
    std::vector<int> p;  // words
    const int base = static_cast<int>(H.prog.size());
    int now = 0, head = -1;
    // an operation of `words` int4 words, within one piece
    auto op = [&](int words, int x, int y) {
      const int at = static_cast<int>(p.size()) / 4;
      if (at % 32 + words > 31) {  // (the piece's last word is its end)
        p.insert(p.end(), {kTfPiece, 0, 0, 0});
        while (p.size() % 128) p.push_back(0);
      }
      head = static_cast<int>(p.size());
      p.insert(p.end(), {x, y, 0, 0});
    };
    auto end_ticks = [&](int upto) {  // barriers until tick `upto`
      if (upto > now && head >= 0) {
        p[head] |= 8;
        ++now;
      }
      if (upto > now) op(1, kTfTicks, upto - now);
      now = upto;
      head = -1;
    };
    auto fill4 = [&]() {
      while (p.size() % 4) p.push_back(0);
    };
    constexpr int kMax = 28;  // words of an operation's list, at most
    // operations over a list, 4 / `per` entries of it to a word
    auto list = [&](int kind, int y, const std::vector<int>& v) {
      for (size_t i = 0; i < v.size(); i += 4 * kMax) {
        const size_t cnt = std::min<size_t>(4 * kMax, v.size() - i), words = (cnt + 3) / 4;
        op(1 + (int)words, kind | (int)words << 5, y);
        p.insert(p.end(), v.begin() + i, v.begin() + i + cnt);
        fill4();
      }
    };
    for (const HostTileSchedule::Op& o : ops[w]) {
      if (o.tick > now) end_ticks(o.tick);
      if (o.task >= N) {
        const int k = o.task - N;
        std::vector<int> in[3];
        for (int i = hp.init_ptr[k] - 1; i < hp.init_ptr[k + 1]; ++i) {
          const bool d = i < hp.init_ptr[k];
          const int* c = kin + 4 * (k + i + 1);
          if (c[1] == 0) continue;
          const int array = c[0] < np ? 0 : c[0] < np + na ? 1 : 2;
          const int index = c[0] - (array == 0 ? 0 : array == 1 ? np : np + na);
          if (index < 0 || index >= 1 << 20) {
            *why = "too many KKT inputs";
            return false;
          }
          in[array].push_back(index | slot[d ? S + k : hp.proc_ptr[k] + init_slot[i]] << 20);
        }
        for (int q = 0; q < 3; ++q) list(kTfLoad, q, in[q]);
      } else if (o.task >= S) {
        const int k = o.task - S, p0 = hp.proc_ptr[k], p1 = hp.proc_ptr[k + 1];
        std::vector<int> raw, zero, constant;
        std::vector<char> has(p1 - p0, 0);
        for (int i = hp.init_ptr[k] - 1; i < hp.init_ptr[k + 1]; ++i) {
          const bool d = i < hp.init_ptr[k];
          const int* c = kin + 4 * (k + i + 1);
          const int s = slot[d ? S + k : p0 + init_slot[i]] * 128;
          // an entry's input is added to 0, d's is taken as it is (adding -0 changes nothing)
          const float zero_sum = d ? -0.0f : 0.0f;
          if (!d) has[init_slot[i]] = 1;
          if (c[1] == 0) constant.insert(constant.end(), {s, d ? c[3] : bits(0.0f + real(c[3]))});
          else if (c[1] == 1) raw.insert(raw.end(), {s, c[2], d || real(c[3]) != 0.0f ? c[3] : bits(0.0f), 0});
          else if (c[1] == 3) raw.insert(raw.end(), {s, bits(-1.0f), bits(zero_sum), 0});
          else raw.insert(raw.end(), {s, c[2], bits(zero_sum), 0});
        }
        for (int e = p0; e < p1; ++e)
          if (!has[e - p0]) zero.push_back(slot[e] * 128);
        list(kTfInputs, 0, raw);
        list(kTfZeros, 0, zero);
        list(kTfConsts, 0, constant);
        if (p0 == p1) {
          op(1, kTfPivot, slot[S + k] * 128);
          H.row_at[k] = base + head + 2;
        }
      } else {
        const int e = o.task, k = row_of[e], words = static_cast<int>(upd[e].size() + 3) / 4;
        const bool last = e + 1 == hp.proc_ptr[k + 1];
        op(1 + last + words,
           static_cast<int>(kTfStep | (last ? 16u : 0u) | (unsigned)words << 5 | (unsigned)slot[S + k] << 21),
           slot[e] * 128 | slot[S + hp.proc_cols[e]] << 18);
        H.step_at[e] = base + head + 2;
        if (last) {
          H.row_at[k] = base + head + 4;
          p.insert(p.end(), {0, 0, 0, 0});
        }
        for (const auto& u : upd[e]) p.push_back(slot[hp.proc_ptr[k] + u.first] * 128 | slot[u.second] << 18);
        fill4();
      }
    }
    if (now < H.ticks) end_ticks(H.ticks);
    p.insert(p.end(), {kTfPiece, 1, 0, 0});
    while (p.size() % 128) p.push_back(0);
    p.resize(p.size() + 3 * 128, 0);  // (the lists are read three pieces ahead)
    H.warp_off.push_back(static_cast<int>(H.prog.size() / 4));
    H.prog.insert(H.prog.end(), p.begin(), p.end());
  }
  return true;
}

}  // namespace wmpc
