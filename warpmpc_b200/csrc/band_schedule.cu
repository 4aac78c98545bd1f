// Host tables of the band form (see band.cuh).
#include <algorithm>
#include <cstring>
#include <numeric>

#include "band.cuh"

namespace wmpc {

size_t band_smem_bytes(int vrows, int yrows, int t4, int n_chunks, int n_items, int chunk_bytes, int ring_bytes,
                       int warps, int stages, int maxima_sets) {
  size_t b = (size_t)(vrows + yrows) * 128 + (size_t)stages * chunk_bytes + (size_t)warps * ring_bytes;
  b += (size_t)((t4 * 4 + 15) / 16) * 16 + (size_t)n_chunks * 24;  // column words, chunk descriptors (chain, producer)
  b += (size_t)((warps * n_items + 1) / 2) * 8;                    // item words
  b += (size_t)maxima_sets * warps * 256;                          // iterate changes and residuals per warp
  b += (size_t)stages * (16 + 4) + 64 + (size_t)warps * 4;         // barriers, tags, counters
  return (b + 127) / 128 * 128;
}

namespace {

int fbits(float v) {
  int i;
  std::memcpy(&i, &v, 4);
  return i;
}

}  // namespace

bool build_band_tables(const HostPattern& hp, const float* rho, const float* rhoinv, const int* rho_type, int n_primal,
                       const float* unscale_by_index, HostBand* out, std::string* why) {
  HostBand& H = *out;
  H = HostBand{};
  const int n = hp.n;
  const std::vector<int>&lp = hp.lp, &li = hp.li;
  for (int c = 0; c < n; ++c)
    for (int e = lp[c]; e < lp[c + 1]; ++e)
      if (li[e] <= c || li[e] >= n || (e > lp[c] && li[e] <= li[e - 1])) {
        *why = "L columns are not ascending";
        return false;
      }
  std::vector<std::vector<std::pair<int, int>>> row(n);  // (column, L entry), ascending
  for (int c = 0; c < n; ++c)
    for (int e = lp[c]; e < lp[c + 1]; ++e) row[li[e]].push_back({c, e});
  // Column classes.  Head: a child is a leaf whose one entry lies in a root's
  // row, a root reads only children and reaches only columns outside the
  // head.  Grow the rest until both hold.
  std::vector<char> rest(n, 0), child(n, 0);
  for (bool more = true; more;) {
    more = false;
    for (int c = 0; c < n; ++c)
      child[c] = !rest[c] && row[c].empty() && lp[c + 1] - lp[c] == 1 && !rest[li[lp[c]]];
    for (int c = 0; c < n; ++c) {
      if (rest[c] || child[c]) continue;
      for (const auto& r : row[c])
        if (!child[r.first]) rest[c] = 1;
      if (rest[c]) more = true;
    }
    for (int c = 0; c < n; ++c) {
      if (rest[c] || child[c]) continue;
      for (int e = lp[c]; e < lp[c + 1]; ++e)
        if (!rest[li[e]]) rest[li[e]] = 1, more = true;
    }
  }
  // The chain takes the rest, except its first columns where a later head
  // column adds to a row they add to (the row's sum runs by ascending
  // column): those make up the *pre-chain*, solved by an item warp.
  int last = -1;
  for (bool more = true; more;) {
    more = false;
    for (int r = 0; r < n; ++r) {
      if (!rest[r] || r <= last) continue;
      int head_last = -1, chain_first = n;
      for (const auto& x : row[r]) {
        if (!rest[x.first] || x.first <= last) head_last = std::max(head_last, x.first);
        else chain_first = std::min(chain_first, x.first);
      }
      if (head_last > chain_first) {
        for (const auto& x : row[r])
          if (rest[x.first] && x.first < head_last && x.first > last) last = x.first, more = true;
      }
    }
  }
  // ... and, while it is short, a leading run that reaches past the window
  // (the chain would wait for those rows' right-hand sides before it starts).
  std::vector<int> all_rest;
  for (int c = 0; c < n; ++c)
    if (rest[c] && c > last) all_rest.push_back(c);
  {
    std::vector<int> at(n, -1);
    for (size_t i = 0; i < all_rest.size(); ++i) at[all_rest[i]] = static_cast<int>(i);
    for (int i = std::min<int>(16, static_cast<int>(all_rest.size()) / 8) - 1; i >= 0; --i) {
      const int c = all_rest[i];
      if (lp[c + 1] > lp[c] && at[li[lp[c + 1] - 1]] - i > 32) {
        last = c;
        break;
      }
    }
  }
  std::vector<int> chain, pre, rank(n, -1), prank(n, -1);
  for (int c = 0; c < n; ++c) {
    if (!rest[c]) continue;
    if (c <= last) {
      prank[c] = static_cast<int>(pre.size());
      pre.push_back(c);
    } else {
      rank[c] = static_cast<int>(chain.size());
      chain.push_back(c);
    }
  }
  if (chain.empty()) {
    *why = "no elimination chain";
    return false;
  }
  if (pre.size() > 64 && pre.size() * 8 > chain.size()) {
    *why = "the elimination chain's start is too long";
    return false;
  }
  H.n = n;
  H.n_prim = n_primal;
  const int T = H.T = static_cast<int>(chain.size());
  const int T4 = H.T4 = (T + 3) / 4 * 4;
  const int n_pre = H.n_pre = static_cast<int>(pre.size());
  // The window: 2 units (8 rows) where no more than a few entries lie past
  // them, else 4 units; entries past the window take the chain warp several
  // times a window entry's work.
  auto far_count = [&](int reach) {
    int far = 0;
    for (int c : chain)
      for (int e = lp[c]; e < lp[c + 1]; ++e) far += rank[li[e]] - rank[c] > reach;
    return far;
  };
  int chain_nnz = 0;
  for (int c : chain) chain_nnz += lp[c + 1] - lp[c];
  H.units = far_count(8) * 50 <= chain_nnz ? 2 : 4;
  const int reach = 4 * H.units;
  if (far_count(reach) * 16 > chain_nnz + 64) {
    *why = "the elimination chain reaches too far";
    return false;
  }
  for (int c = 0; c < n; ++c)
    if (!rest[c] && !child[c] && lp[c + 1] - lp[c] > 60 - kBandChildren) {
      *why = "a head column has too many entries";
      return false;
    }
  for (int c : pre)
    if (lp[c + 1] - lp[c] > 60) {
      *why = "a pre-chain column has too many entries";
      return false;
    }
  auto kind_of = [&](int k) {
    const int orig = hp.p[k], r = orig - n_primal;
    return orig < n_primal ? 0 : 1 | ((rho_type ? rho_type[r] : 0) + 1) << 1;
  };
  auto consts_of = [&](int k, std::vector<int>* v) {
    const int orig = hp.p[k], r = orig - n_primal;
    const bool cons = orig >= n_primal;
    v->insert(v->end(), {cons ? fbits(rho[r]) : 0, cons ? fbits(rhoinv[r]) : 0,
                         fbits(unscale_by_index ? unscale_by_index[orig] : 1.0f), cons ? r * 32 : 0});
  };
  auto par_floats = [&](int k) { return hp.p[k] >= n_primal ? 64 : 32; };
  H.lpos.assign(std::max(hp.nnz_l, 1), -1);
  H.lpos2.assign(std::max(hp.nnz_l, 1), -1);
  H.dpos.assign(n, -1);
  H.iter_off.assign(n, -1);
  H.param_off.assign(n, -1);
  int off = 0;
  // ---- chain chunks of about 9 KB ----
  H.chunk_cols = H.units == 2 ? 8 : 4;
  H.n_chunks = (T4 + H.chunk_cols - 1) / H.chunk_cols;
  H.col_word.assign(T4, 0);
  for (int ch = 0; ch < H.n_chunks; ++ch) {
    const int t0 = ch * H.chunk_cols, t1 = std::min(t0 + H.chunk_cols, T4), start = off;
    int unit = 0, last = std::min(T, t1 + reach);
    std::vector<std::pair<int, int>> far;  // (column in the chunk, L entry)
    for (int t = t0; t < t1; ++t) {
      int near_last = 0;
      const int c = t < T ? chain[t] : -1;
      for (int e = c < 0 ? 0 : lp[c]; c >= 0 && e < lp[c + 1]; ++e) {
        const int d = rank[li[e]] - t;
        if (d <= reach) near_last = d; else far.push_back({t - t0, e});
      }
      const int u = near_last > 4 * (H.units - 1) ? H.units : H.units - 1, base = start + unit * 128;
      std::vector<char> used(4 * u, 0);
      for (int e = c < 0 ? 0 : lp[c]; c >= 0 && e < lp[c + 1]; ++e) {
        const int d = rank[li[e]] - t;
        if (d > reach) continue;
        used[d - 1] = 1;
        H.lpos[e] = base + ((d - 1) >> 2) * 128 + ((d - 1) & 3);
      }
      for (int i = 0; i < 4 * u; ++i)
        if (!used[i]) H.pad.push_back(base + (i >> 2) * 128 + (i & 3));
      H.col_word[t] = (u == H.units ? 1 : 0) | unit << 1;
      unit += u;
    }
    H.far_ptr.push_back(static_cast<int>(H.far.size() / 4));
    for (size_t i = 0; i < far.size(); ++i) {
      const int e = far[i].second, at = (unit + static_cast<int>(i >> 2)) * 128 + static_cast<int>(i & 3);
      H.lpos[e] = start + at;
      H.far.insert(H.far.end(), {far[i].first, rank[li[e]] * 128, at * 4, 0});
      last = std::max(last, rank[li[e]] + 1);
    }
    unit += static_cast<int>(far.size() + 3) / 4;
    if (far.size() > 255) {
      *why = "too many far entries in one chunk";
      return false;
    }
    off = start + unit * 128;
    for (int t = t0; t < std::min(t1, T); ++t) {
      H.dpos[chain[t]] = off;
      off += 32;
    }
    if (t1 > T) {  // D^-1 of the columns past T: zero (one unit holds them all)
      for (int i = 0; i < 4; ++i) H.pad.push_back(off + i);
      off += 128;
    }
    H.chunk.insert(H.chunk.end(), {start, unit * 512, (t1 - t0) | static_cast<int>(far.size()) << 8, last});
    H.chunk_bytes = std::max(H.chunk_bytes, (off - start) * 4);
  }
  // ---- subtrees ----
  // backward chunks that must be done before a column's chain rows are final
  auto need_of = [&](int c) {
    int need = 0;
    for (int e = lp[c]; e < lp[c + 1]; ++e)
      if (rank[li[e]] >= 0) need = std::max(need, H.n_chunks - rank[li[e]] / H.chunk_cols);
    return need;
  };
  auto uses_pre = [&](int c) {
    for (int e = lp[c]; e < lp[c + 1]; ++e)
      if (prank[li[e]] >= 0) return true;
    return false;
  };
  int pre_need = 0;
  for (int c : pre) pre_need = std::max(pre_need, need_of(c));
  struct Sub {
    int root, need;
    std::vector<int> child;
  };
  std::vector<Sub> subs;
  std::vector<int> sub_of(n, -1);
  for (int c = 0; c < n; ++c)
    if (!rest[c] && !child[c]) {
      sub_of[c] = static_cast<int>(subs.size());
      // (after the pre-chain, where it is read: its own chunks and some slack; one chunk
      // where it reads no chain row: the zero row of its padding and of its children's
      // slots is written in the first F phase, which the chain waits for)
      subs.push_back(
          Sub{c, uses_pre(c) ? std::min(H.n_chunks, std::max(need_of(c), pre_need + 1)) : std::max(need_of(c), 1), {}});
    }
  for (int c = 0; c < n; ++c)
    if (child[c]) subs[sub_of[li[lp[c]]]].child.push_back(c);
  H.nb = static_cast<int>(subs.size());
  H.n_yr = H.nb + n_pre;
  std::vector<int> order(subs.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {  // (one after the other go to different warps)
    if (subs[a].need != subs[b].need) return subs[a].need < subs[b].need;
    return lp[subs[a].root + 1] - lp[subs[a].root] > lp[subs[b].root + 1] - lp[subs[b].root];
  });
  std::vector<int> yr_of(n, -1);
  for (size_t i = 0; i < order.size(); ++i) yr_of[subs[order[i]].root] = static_cast<int>(i);
  for (int c : pre) yr_of[c] = H.nb + prank[c];
  const int vzero = band_vzero(T4, H.units);
  auto v_of = [&](int c) { return rank[c] >= 0 ? rank[c] : vzero + 1 + prank[c]; };
  if (H.n_chunks >= kBandUsesPre) {
    *why = "too many chunks";
    return false;
  }
  // an item is opened with its record's size, placed at `off`, and closed with
  // its record
  auto row_floats = [&](int words) { return (words + 31) / 32 * 32; };
  bool fits = true;
  auto open_item = [&](int rec_words) -> int {  // stream offset of the item
    const int at = off;
    off += row_floats(rec_words);
    return at;
  };
  auto close_item = [&](int at, std::vector<int> rec) {
    rec[0] |= row_floats((int)rec.size()) / 32 << 27;
    rec.resize(row_floats((int)rec.size()), 0);
    for (size_t i = 0; i < rec.size(); i += 32) H.rec_off.push_back(at + (int)i);
    H.rec.insert(H.rec.end(), rec.begin(), rec.end());
    const int rows = (off - at) / 32;
    if (at / 32 >= 1 << 22 || rows >= 1 << 10) fits = false;
    H.item.push_back(static_cast<int>((unsigned)(at / 32) | (unsigned)rows << 22));
    H.item_bytes = std::max(H.item_bytes, rows * 128);
  };
  // a column's entries in its units (`keep` last slots are not padding), their rows appended to the record
  auto entry_slots = [&](int c, int base, int units, int keep, std::vector<int>* rec) {
    const int cnt = lp[c + 1] - lp[c];
    for (int e = 0; e < units * 4; ++e) {
      const int pos = base + (e >> 2) * 128 + (e & 3);
      if (e < cnt) H.lpos[lp[c] + e] = pos;
      else if (e < units * 4 - keep) H.pad.push_back(pos);
      rec->push_back((e < cnt ? v_of(li[lp[c] + e]) : vzero) * 128);
    }
  };
  auto place_index = [&](int k) {  // parameters, then iterate
    H.param_off[hp.p[k]] = off;
    H.iter_off[hp.p[k]] = off + par_floats(k);
    off += 2 * par_floats(k);
  };
  // the pre-chain's columns, last first: solved here, their rows' updates are F items
  for (int i = n_pre - 1; i >= 0; --i) {
    const int c = pre[i], units = (lp[c + 1] - lp[c] + 3) / 4;
    const int at = open_item(kBandRecB + 4 * units);
    std::vector<int> rec{units, yr_of[c] * 128, need_of(c), v_of(c) * 128};
    rec.resize(kBandRecB, 0);
    entry_slots(c, off, units, 0, &rec);
    off += units * 128;
    H.dpos[c] = off;
    off += 32;
    close_item(at, rec);
  }
  for (int so : order) {
    const Sub& s = subs[so];
    const int c = s.root, nc = static_cast<int>(s.child.size());
    if (nc > kBandChildren) {
      *why = "a head column has too many children";
      return false;
    }
    const int units = (lp[c + 1] - lp[c] + nc + 3) / 4;
    const int at = open_item(kBandRecB + 4 * units), base = off;
    off += units * 128;
    int kinds = kind_of(c) << 8;
    std::vector<int> rec{0, yr_of[c] * 128, s.need | (uses_pre(c) ? kBandUsesPre : 0), off};
    auto place = [&](int col) {
      H.dpos[col] = off;
      off += 32;
      place_index(col);
      consts_of(col, &rec);
    };
    place(c);
    for (int i = 0; i < nc; ++i) {
      const int slot = units * 4 - 1 - i;
      H.lpos[lp[s.child[i]]] = base + (slot >> 2) * 128 + (slot & 3);
      kinds |= kind_of(s.child[i]) << (12 + 4 * i);
      place(s.child[i]);
    }
    rec[0] = units | nc << 4 | kinds;
    rec.resize(kBandRecB, 0);
    entry_slots(c, base, units, nc, &rec);
    close_item(at, rec);
  }
  // ---- F items: the pre-chain's rows, then the chain's ----
  for (int pass = 0; pass < 2; ++pass) {
    for (int k : pass == 0 ? pre : chain) {
      std::vector<std::pair<int, int>> ent;  // head and pre-chain entries, ascending column
      for (const auto& x : row[k])
        if (rank[x.first] < 0) ent.push_back(x);
      const int cnt = static_cast<int>(ent.size()), units = (cnt + 3) / 4;
      if (units > 60) {
        *why = "a row has too many head entries";
        return false;
      }
      const int at = open_item(kBandRecF + 4 * units), base = off;
      off += units * 128;
      std::vector<int> rec{0, v_of(k) * 128, pass == 0 ? yr_of[k] * 128 : -1, off};
      consts_of(k, &rec);
      bool pre_used = false;
      for (int e = 0; e < units * 4; ++e) {
        const int pos = base + (e >> 2) * 128 + (e & 3);
        if (e < cnt) {
          H.lpos2[ent[e].second] = pos;
          pre_used = pre_used || prank[ent[e].first] >= 0;
        } else {
          H.pad.push_back(pos);
        }
        rec.push_back((e < cnt ? yr_of[ent[e].first] : H.n_yr) * 128);
      }
      rec[0] = units | kind_of(k) << 8 | (pre_used ? kBandUsesPre : 0);
      place_index(k);
      close_item(at, rec);
    }
  }
  if (!fits) {
    *why = "an item is too large";
    return false;
  }
  const int scratch = off;  // where entries without a copy write theirs
  off += 128;
  for (int e = 0; e < hp.nnz_l; ++e)
    if (H.lpos2[e] < 0) H.lpos2[e] = scratch;
  H.blen = off;
  const int warps = H.units > 2 ? kBandWideWarps : kBandWarps;
  if (band_smem_bytes(band_vrows(T4, H.units, n_pre), H.n_yr + 1, T4, H.n_chunks, band_items(n_pre, H.nb, T, warps),
                      H.chunk_bytes, H.item_bytes, warps, kBandStages, band_maxima_sets(T, warps)) >
      (size_t)kMaxSmemBytes) {
    *why = "band work vectors do not fit in shared memory";
    return false;
  }
  // every word the kernels use as an address stays inside its array
  for (int e = 0; e < hp.nnz_l; ++e)
    if (H.lpos[e] < 0 || H.lpos[e] + 124 >= H.blen || H.lpos2[e] < 0 || H.lpos2[e] + 124 >= H.blen) {
      *why = "band L position out of range";
      return false;
    }
  for (int k = 0; k < n; ++k)
    if (H.dpos[k] < 0 || H.dpos[k] + 32 > H.blen || H.iter_off[k] < 0 || H.param_off[k] < 0 ||
        H.iter_off[k] + 32 > H.blen || H.param_off[k] + 32 > H.blen) {
      *why = "band record out of range";
      return false;
    }
  return true;
}

}  // namespace wmpc
