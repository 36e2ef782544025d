// Symbolic elimination of the parts (host): the order, N+(v) of every inner
// vertex, and the levels that may be processed at once.  See fap_elim.h.
#include "fap_elim.h"

#include <algorithm>
#include <atomic>
#include <thread>

namespace fapb {
namespace {

struct PartPlan {
  bool ok = false;
  int32_t b = 0, boff = 0;
  std::vector<int32_t> loc, inv, eptr, ecol, w0, w0b, lev;
  std::vector<ElimUnit> units;
  std::vector<int32_t> glev, rows8;
  std::vector<uint16_t> list;
  std::vector<int32_t> sloc;
  std::vector<ElimChunk> chunks;
  int32_t stream16 = 0;
  int64_t group_work = 0;
};

// Least-degree elimination of one part on bitset rows: joining v's
// neighbours is an OR of v's row into each of theirs.  Half the depth of the
// neighbourhoods eliminated so far counts as degree: the sweeps are bound by
// their levels, and pendant paths and chains are then taken every other
// vertex instead of end to end (road114k: 17 levels instead of 53 with 1.46
// entries per vertex instead of 1.36; a 256 x 256 grid 101 instead of 113).
void eliminate(const ElimGraph &g, int32_t inf, bool directed, PartPlan *out) {
  const int32_t s = g.s, b = g.b;
  const int W = (s + 63) / 64;
  std::vector<uint64_t> A((size_t)s * W, 0);
  for (int32_t i = 0; i < s; i++)
    for (int32_t e = g.ptr[i]; e < g.ptr[i + 1]; e++) {
      const int32_t j = g.adj[e];
      A[(size_t)i * W + j / 64] |= uint64_t(1) << (j % 64);
      A[(size_t)j * W + i / 64] |= uint64_t(1) << (i % 64);
    }
  std::vector<int32_t> deg(s), up(s, 0);
  for (int32_t i = 0; i < s; i++) {
    int32_t d = 0;
    for (int w = 0; w < W; w++) d += __builtin_popcountll(A[(size_t)i * W + w]);
    deg[i] = d;
  }
  // buckets by key; entries of outdated keys are skipped
  auto key = [&](int32_t v) { return 2 * deg[v] + up[v]; };
  std::vector<std::vector<int32_t>> bucket;
  int32_t low = 0;
  auto push = [&](int32_t v) {
    const int32_t k = key(v);
    if ((size_t)k >= bucket.size()) bucket.resize(k + 1);
    bucket[k].push_back(v);
    low = std::min(low, k);
  };
  for (int32_t i = b; i < s; i++) push(i);
  std::vector<int32_t> nptr(s, 0), ncnt(s, 0), nbr;  // N+ of the eliminated vertices
  std::vector<int> words;
  std::vector<char> gone(s, 0);
  std::vector<int32_t> order;
  order.reserve(std::max(0, s - b));
  const size_t limit = (size_t)((int64_t)s * std::max(s, 256) / kElimDense);
  while ((int32_t)order.size() < s - b) {
    while (bucket[low].empty()) low++;
    const int32_t v = bucket[low].back();
    bucket[low].pop_back();
    if (gone[v] || key(v) != low) continue;
    gone[v] = 1;
    order.push_back(v);
    nptr[v] = (int32_t)nbr.size();
    const uint64_t *rv = &A[(size_t)v * W];
    for (int w = 0; w < W; w++)
      for (uint64_t x = rv[w]; x != 0; x &= x - 1) nbr.push_back(w * 64 + __builtin_ctzll(x));
    ncnt[v] = (int32_t)nbr.size() - nptr[v];
    if (nbr.size() > limit) return;
    words.clear();  // (the neighbours sit in a few words of the row)
    for (int w = 0; w < W; w++)
      if (rv[w] != 0) words.push_back(w);
    for (int32_t i = 0; i < ncnt[v]; i++) {
      const int32_t u = nbr[nptr[v] + i];
      uint64_t *ru = &A[(size_t)u * W];
      int32_t d = 0;
      for (int w : words) {
        d += __builtin_popcountll(rv[w] & ~ru[w]);
        ru[w] |= rv[w];
      }
      ru[v / 64] &= ~(uint64_t(1) << (v % 64));
      ru[u / 64] &= ~(uint64_t(1) << (u % 64));
      if (u < b) continue;
      deg[u] += d - 2;  // (u's own bit came with rv, v is gone)
      up[u] = std::max(up[u], up[v] + 1);
      push(u);
    }
  }
  const int64_t nnz = (int64_t)nbr.size();
  // levels: the depths, highest first; within a level in elimination order
  int32_t top = -1;
  for (int32_t v : order) top = std::max(top, up[v]);
  std::vector<int32_t> cnt(top + 2, 0);
  for (int32_t v : order) cnt[top - up[v] + 1]++;
  out->lev.assign(top + 2, b);
  for (int32_t l = 0; l <= top; l++) out->lev[l + 1] = out->lev[l] + cnt[l + 1];
  std::vector<int32_t> fill(out->lev.begin(), out->lev.end());
  out->loc.resize(s);
  out->inv.resize(s);
  for (int32_t i = 0; i < b; i++) out->loc[i] = i;
  for (auto it = order.rbegin(); it != order.rend(); ++it) out->loc[fill[top - up[*it]]++] = *it;
  for (int32_t e = 0; e < s; e++) out->inv[out->loc[e]] = e;
  out->eptr.assign(s + 1, 0);
  for (int32_t e = 0; e < s; e++)
    out->eptr[e + 1] = out->eptr[e] + (e < b ? 0 : ncnt[out->loc[e]]);
  out->ecol.resize(nnz);
  out->w0.assign(nnz, inf);
  if (directed) out->w0b.assign(nnz, inf);
  // N+ in descending plan numbers: every u appends itself to the lists that
  // hold it, the last u first (sorting list by list took three times as long)
  std::vector<int32_t> rptr(s + 1, 0), rev(nnz), at(s);
  for (int32_t u : nbr) rptr[u + 1]++;
  for (int32_t u = 0; u < s; u++) {
    rptr[u + 1] += rptr[u];
    at[u] = rptr[u];
  }
  for (int32_t v : order)
    for (int32_t i = nptr[v]; i < nptr[v] + ncnt[v]; i++) rev[at[nbr[i]]++] = out->inv[v];
  std::copy(out->eptr.begin(), out->eptr.end() - 1, at.begin());  // (by plan number from here on)
  for (int32_t e = s - 1; e >= 0; e--) {
    const int32_t u = out->loc[e];
    for (int32_t i = rptr[u]; i < rptr[u + 1]; i++) out->ecol[at[rev[i]]++] = e;
  }
  if (!g.w.empty())
    for (int32_t i = 0; i < s; i++)
      for (int32_t a = g.ptr[i]; a < g.ptr[i + 1]; a++) {
        const int32_t x = out->inv[i], y = out->inv[g.adj[a]], v = std::max(x, y), u = std::min(x, y);
        if (v < b) continue;
        const int32_t *c = out->ecol.data() + out->eptr[v], *end = out->ecol.data() + out->eptr[v + 1];
        const auto at = std::lower_bound(c, end, u, std::greater<int32_t>()) - out->ecol.data();
        if (x > y) out->w0[at] = g.w[a];
        else if (directed) out->w0b[at] = g.w[a];
      }
  out->ok = true;
}

// Separator groups from the elimination order (plan numbers descending).  A
// group's cost is its chunks of four rows times its list, plus kChunkCost
// entries' worth for storing the rows.
constexpr int64_t kChunkCost = 6;

void group_rows(PartPlan *q) {
  const int32_t s = (int32_t)q->loc.size(), b = q->b;
  auto deg = [&](int32_t v) { return q->eptr[v + 1] - q->eptr[v]; };
  auto cost = [&](int64_t g, int64_t u) { return (g + 3) / 4 * (u + kChunkCost); };
  std::vector<int32_t> size(s, 0), into(s, -1), par(s, -1);
  std::vector<std::vector<int32_t>> child(s);
  for (int32_t v = s - 1; v >= b; v--) {
    size[v] = 1;
    for (int32_t c : child[v])
      if (cost(size[v] + size[c], deg(v)) <= cost(size[v], deg(v)) + cost(size[c], deg(c))) {
        size[v] += size[c];
        into[c] = v;
      }
    if (deg(v) > 0 && q->ecol[q->eptr[v]] >= b) {
      par[v] = q->ecol[q->eptr[v]];
      child[par[v]].push_back(v);
    }
  }
  std::vector<int32_t> rep(s, -1), lev(s, -1);
  std::vector<std::vector<int32_t>> rows(s);
  int32_t nlev = 0;
  for (int32_t v = b; v < s; v++) {
    rep[v] = into[v] >= 0 ? rep[into[v]] : v;
    rows[rep[v]].push_back(v);
    if (rep[v] == v) {
      lev[v] = par[v] >= 0 ? lev[rep[par[v]]] + 1 : 0;
      nlev = std::max(nlev, lev[v] + 1);
    }
  }
  // slots: the boundary vertices and every row that a list names
  std::vector<int32_t> slot(s, -1);
  for (int32_t v = b; v < s; v++)
    if (rep[v] == v)
      for (int32_t i = q->eptr[v]; i < q->eptr[v + 1]; i++) slot[q->ecol[i]] = 0;
  for (int32_t v = 0; v < s; v++)
    if (v < b || slot[v] == 0) {
      slot[v] = (int32_t)q->sloc.size();
      q->sloc.push_back(q->loc[v]);
    }
  std::vector<std::vector<ElimUnit>> units(nlev);
  for (int32_t v = b; v < s; v++) {
    if (rep[v] != v) continue;
    const int32_t list = (int32_t)q->list.size(), nu = (deg(v) + 3) / 4 * 4;
    for (int32_t i = 0; i < nu; i++)
      q->list.push_back((uint16_t)slot[q->ecol[q->eptr[v] + std::min(i, deg(v) - 1)]]);
    for (size_t r = 0; r < rows[v].size(); r += kElimUnitRows) {
      const int32_t k = (int32_t)std::min<size_t>(kElimUnitRows, rows[v].size() - r);
      const bool wide = k > 4;
      units[lev[v]].push_back(ElimUnit{(int32_t)q->rows8.size() / 2, list, nu | (wide ? kElimWide : 0), 0, 0, 0});
      for (int32_t i = 0; i < kElimUnitRows; i++) {
        q->rows8.push_back(i < k ? slot[rows[v][r + i]] : -1);
        q->rows8.push_back(i < k ? q->loc[rows[v][r + i]] : -1);
      }
      q->group_work += (int64_t)nu * (wide ? 8 : 4);
    }
  }
  q->glev.push_back(0);
  for (auto &u : units) {  // longest first: the last units of a level are short
    std::stable_sort(u.begin(), u.end(),
                     [](const ElimUnit &x, const ElimUnit &y) { return elim_body16(x.nu) > elim_body16(y.nu); });
    for (size_t i = 0; i < u.size();) {
      size_t k = i;
      int32_t bodies = 0;
      while (k < u.size() && (k == i || bodies + elim_body16(u[k].nu) + (int32_t)(k - i + 2) / 2 <= kElimChunk16))
        bodies += elim_body16(u[k++].nu);
      const int32_t off = q->stream16, heads = (int32_t)(k - i + 1) / 2;
      q->chunks.push_back(ElimChunk{off, heads + bodies, (int32_t)(k - i), 0});
      int32_t body = off + heads;
      for (size_t j = i; j < k; j++) {
        u[j].head = 2 * off + (int32_t)(j - i);
        u[j].body = body;
        u[j].chunk = off;
        body += elim_body16(u[j].nu);
      }
      q->stream16 = body;
      i = k;
    }
    q->units.insert(q->units.end(), u.begin(), u.end());
    q->glev.push_back((int32_t)q->units.size());
  }
}

}  // namespace

namespace {
// work() on up to `threads` threads, this one among them.
template <typename F>
void run_threads(int threads, F work) {
  std::vector<std::thread> pool;
  try {
    for (int t = 1; t < threads; t++) pool.emplace_back(work);
  } catch (...) {  // fewer threads than asked for
  }
  work();
  for (std::thread &t : pool) t.join();
}

template <typename T>
void put(PlanArray<T> *to, size_t at, const std::vector<T> &from) {
  std::copy(from.begin(), from.end(), to->data() + at);
}
}  // namespace

void elim_build(int nparts, const std::function<void(int, ElimGraph *)> &graph, int threads, int32_t inf,
                bool directed, bool groups, ElimPlan *out) {
  *out = ElimPlan{};
  const int K = nparts;
  std::vector<PartPlan> pp(K);
  std::atomic<int> next{0};
  std::atomic<bool> dense{false};
  std::atomic<bool> failed{false};  // an allocation failed: no plan
  threads = std::max(1, std::min(threads, K));
  run_threads(threads, [&] {
    try {
      for (int p = next++; p < K && !dense; p = next++) {
        ElimGraph g;
        graph(p, &g);
        pp[p].boff = g.boff;
        pp[p].b = g.b;
        if (g.s <= kElimMaxS) eliminate(g, inf, directed, &pp[p]);
        if (!pp[p].ok) dense = true;
        else if (groups && g.b > kThinBoundary) group_rows(&pp[p]);  // (the others take the thin merge)
      }
    } catch (...) {
      failed = true;
      dense = true;
    }
  });
  if (dense || failed) return;
  // The parts' places in the plan's arrays, then the copies.
  size_t nv = 0, ne = 0, np = 0, nl = 0, ng = 0, nu = 0, nr = 0, ns = 0, ni = 0, nc = 0;
  std::vector<int32_t> unit0(K), rows0(K), list0(K);
  for (int p = 0; p < K; p++) {
    const PartPlan &q = pp[p];
    ElimPart d{};
    d.s = (int32_t)q.loc.size();
    d.b = q.b;
    d.boff = q.boff;
    d.voff = (int32_t)nv;
    d.eptr_off = (int32_t)np;
    d.ent_off = (int32_t)ne;
    d.nent = (int32_t)q.ecol.size();
    d.lev_off = (int32_t)nl;
    d.nlev = (int32_t)q.lev.size() - 1;
    d.glev_off = (int32_t)ng;
    d.gnlev = std::max(0, (int32_t)q.glev.size() - 1);
    d.stream_off = (int32_t)out->stream16;
    d.chunk_off = (int32_t)nc;
    d.nchunks = (int32_t)q.chunks.size();
    d.nslots = (int32_t)q.sloc.size();
    d.sloc_off = (int32_t)ns;
    unit0[p] = (int32_t)nu;
    rows0[p] = (int32_t)(nr / 2);
    list0[p] = (int32_t)ni;
    nv += q.loc.size();
    np += q.eptr.size();
    ne += q.ecol.size();
    nl += q.lev.size();
    ng += q.glev.size();
    nu += q.units.size();
    nr += q.rows8.size();
    ns += q.sloc.size();
    ni += q.list.size();
    nc += q.chunks.size();
    for (const ElimChunk &c : q.chunks) out->max_chunk16 = std::max(out->max_chunk16, c.n16);
    out->max_chunks = std::max(out->max_chunks, d.nchunks);
    out->stream16 += q.stream16;
    out->group_work.push_back(q.group_work);
    out->max_s = std::max(out->max_s, d.s);
    out->max_nent = std::max(out->max_nent, d.nent);
    out->max_nlev = std::max(out->max_nlev, d.nlev);
    out->parts.push_back(d);
  }
  out->nent = (int64_t)ne;
  if (out->nent >= INT32_MAX / 2 || out->stream16 >= INT32_MAX / 2) return;
  out->loc.make(nv);
  out->inv.make(nv);
  out->eptr.make(np);
  out->ecol.make(ne);
  out->eend.make(ne);
  out->w0.make(ne);
  out->w0b.make(directed ? ne : 0);
  out->lev.make(nl);
  out->units.make(nu);
  out->glev.make(ng);
  out->rows8.make(nr);
  out->list.make(ni);
  out->sloc.make(ns);
  out->chunks.make(nc);
  next = 0;
  // (small plans: a thread costs more than its share of the copies)
  run_threads((int)std::min<size_t>(threads, 1 + ne / 16384), [&] {
    for (int p = next++; p < K; p = next++) {
      const PartPlan &q = pp[p];
      const ElimPart &d = out->parts[p];
      put(&out->loc, d.voff, q.loc);
      put(&out->inv, d.voff, q.inv);
      put(&out->eptr, d.eptr_off, q.eptr);
      put(&out->ecol, d.ent_off, q.ecol);
      put(&out->w0, d.ent_off, q.w0);
      if (directed) put(&out->w0b, d.ent_off, q.w0b);
      for (int32_t e = 0; e < d.s; e++)
        std::fill(out->eend.data() + d.ent_off + q.eptr[e], out->eend.data() + d.ent_off + q.eptr[e + 1], q.eptr[e + 1]);
      put(&out->lev, d.lev_off, q.lev);
      for (size_t i = 0; i < q.units.size(); i++) {
        ElimUnit u = q.units[i];
        u.rows += rows0[p];
        u.list += list0[p];
        out->units[unit0[p] + i] = u;
      }
      for (size_t i = 0; i < q.glev.size(); i++) out->glev[d.glev_off + i] = unit0[p] + q.glev[i];
      put(&out->rows8, 2 * (size_t)rows0[p], q.rows8);
      put(&out->list, list0[p], q.list);
      put(&out->sloc, d.sloc_off, q.sloc);
      put(&out->chunks, d.chunk_off, q.chunks);
    }
  });
  out->ok = true;
}

void elim_offsets(int64_t ld, ElimPlan *plan) {
  for (const ElimPart &d : plan->parts)
    for (int32_t v = d.b; v < d.s; v++)
      for (int32_t e = plan->eptr[d.eptr_off + v]; e < plan->eptr[d.eptr_off + v + 1]; e++)
        plan->w0[d.ent_off + e] =
            (int32_t)(plan->loc[d.voff + v] * ld + plan->loc[d.voff + plan->ecol[d.ent_off + e]]);
}

}  // namespace fapb
