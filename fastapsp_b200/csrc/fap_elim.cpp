// Symbolic elimination of the parts (host): the order, N+(v) of every inner
// vertex, and the levels that may be processed at once.  See fap_elim.h.
#include "fap_elim.h"

#include <algorithm>
#include <atomic>
#include <thread>

namespace fapb {
namespace {

constexpr int32_t kInf = 100000000;

struct PartPlan {
  bool ok = false;
  int32_t b = 0, boff = 0;
  std::vector<int32_t> loc, inv, eptr, ecol, w0, lev;
};

// Least-degree elimination of one part on bitset rows: joining v's
// neighbours is an OR of v's row into each of theirs.  Half the depth of the
// neighbourhoods eliminated so far counts as degree: the sweeps are bound by
// their levels, and pendant paths and chains are then taken every other
// vertex instead of end to end (road114k: 17 levels instead of 53 with 1.46
// entries per vertex instead of 1.36; a 256 x 256 grid 101 instead of 113).
void eliminate(const ElimGraph &g, PartPlan *out) {
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
    for (int32_t i = 0; i < ncnt[v]; i++) {
      const int32_t u = nbr[nptr[v] + i];
      uint64_t *ru = &A[(size_t)u * W];
      int32_t d = 0;
      for (int w = 0; w < W; w++) d += __builtin_popcountll(ru[w] |= rv[w]);
      ru[v / 64] &= ~(uint64_t(1) << (v % 64));
      ru[u / 64] &= ~(uint64_t(1) << (u % 64));
      if (u < b) continue;
      deg[u] = d - 2;  // (v and u itself, both set by rv or before)
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
  out->w0.assign(nnz, kInf);
  for (int32_t e = b; e < s; e++) {
    const int32_t v = out->loc[e];
    int32_t *c = &out->ecol[out->eptr[e]];
    int32_t k = 0;
    for (int32_t i = 0; i < ncnt[v]; i++) c[k++] = out->inv[nbr[nptr[v] + i]];
    std::sort(c, c + k, std::greater<int32_t>());
    if (g.w.empty()) continue;
    for (int32_t a = g.ptr[v]; a < g.ptr[v + 1]; a++) {
      const int32_t u = out->inv[g.adj[a]];
      int32_t *p = std::lower_bound(c, c + k, u, std::greater<int32_t>());
      if (p != c + k && *p == u) {
        int32_t &x = out->w0[out->eptr[e] + (p - c)];
        x = std::min(x, g.w[a]);
      }
    }
  }
  out->ok = true;
}

}  // namespace

void elim_build(int nparts, const std::function<void(int, ElimGraph *)> &graph, int threads, ElimPlan *out) {
  *out = ElimPlan{};
  const int K = nparts;
  std::vector<PartPlan> pp(K);
  std::atomic<int> next{0};
  std::atomic<bool> dense{false};
  std::atomic<bool> failed{false};  // an allocation failed: no plan
  auto work = [&] {
    try {
      for (int p = next++; p < K && !dense; p = next++) {
        ElimGraph g;
        graph(p, &g);
        pp[p].boff = g.boff;
        pp[p].b = g.b;
        if (g.s <= kElimMaxS) eliminate(g, &pp[p]);
        if (!pp[p].ok) dense = true;
      }
    } catch (...) {
      failed = true;
      dense = true;
    }
  };
  const int nt = std::max(1, std::min(threads, K));
  std::vector<std::thread> pool;
  try {
    for (int t = 1; t < nt; t++) pool.emplace_back(work);
  } catch (...) {  // fewer threads than asked for
  }
  work();
  for (std::thread &t : pool) t.join();
  if (dense || failed) return;
  size_t nv = 0, ne = 0;
  for (const PartPlan &q : pp) {
    nv += q.loc.size();
    ne += q.ecol.size();
  }
  out->loc.reserve(nv);
  out->inv.reserve(nv);
  out->eptr.reserve(nv + K);
  for (auto *a : {&out->ecol, &out->eend, &out->w0}) a->reserve(ne);
  for (int p = 0; p < K; p++) {
    const PartPlan &q = pp[p];
    ElimPart d{};
    d.s = (int32_t)q.loc.size();
    d.b = q.b;
    d.boff = q.boff;
    d.voff = (int32_t)out->loc.size();
    d.eptr_off = (int32_t)out->eptr.size();
    d.ent_off = (int32_t)out->ecol.size();
    d.nent = (int32_t)q.ecol.size();
    d.lev_off = (int32_t)out->lev.size();
    d.nlev = (int32_t)q.lev.size() - 1;
    out->parts.push_back(d);
    out->loc.insert(out->loc.end(), q.loc.begin(), q.loc.end());
    out->inv.insert(out->inv.end(), q.inv.begin(), q.inv.end());
    out->eptr.insert(out->eptr.end(), q.eptr.begin(), q.eptr.end());
    out->ecol.insert(out->ecol.end(), q.ecol.begin(), q.ecol.end());
    out->w0.insert(out->w0.end(), q.w0.begin(), q.w0.end());
    out->lev.insert(out->lev.end(), q.lev.begin(), q.lev.end());
    for (int32_t e = 0; e < d.s; e++)
      out->eend.insert(out->eend.end(), q.eptr[e + 1] - q.eptr[e], q.eptr[e + 1]);
    out->max_s = std::max(out->max_s, d.s);
    out->max_b = std::max(out->max_b, d.b);
    out->max_nent = std::max(out->max_nent, d.nent);
    out->max_nlev = std::max(out->max_nlev, d.nlev);
  }
  out->nent = (int64_t)out->ecol.size();
  out->ok = out->nent < INT32_MAX / 2;
}

void elim_offsets(int64_t ld, ElimPlan *plan) {
  for (const ElimPart &d : plan->parts)
    for (int32_t v = d.b; v < d.s; v++)
      for (int32_t e = plan->eptr[d.eptr_off + v]; e < plan->eptr[d.eptr_off + v + 1]; e++)
        plan->w0[d.ent_off + e] =
            (int32_t)(plan->loc[d.voff + v] * ld + plan->loc[d.voff + plan->ecol[d.ent_off + e]]);
}

}  // namespace fapb
