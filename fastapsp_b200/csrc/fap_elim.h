// Vertex elimination inside the parts of an undirected int32 graph: the host
// plan (fap_elim.cpp) and the launchers of its kernels (fap_elim.cu).
// Internal, not installed.
//
// Every part's inner vertices are eliminated one after the other (least
// remaining degree first, boundary vertices never).  Eliminating v joins the
// vertices N+(v) it is still adjacent to, so that every path from v to a
// vertex not eliminated before v leaves through N+(v): with W(v, u) the
// shortest path from v to u through vertices eliminated earlier,
//   D[v][x] = min over u in N+(v) of W(v, u) + D[u][x]
// for every x that is not eliminated before v.  Sums and minima of int32 are
// exact, so the values are those of Floyd-Warshall (float32 sums associate
// differently, with fewer roundings on a path than edge after edge).  Directed
// parts keep both weights of an entry, W(v, u) and W(u, v).  On road-shaped parts
// N+(v) holds 1.4 vertices on average (a part of 830 vertices: 1,300
// relaxations per column instead of 830^2), on grid parts about 20.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <memory>
#include <vector>

#include "fap_internal.h"

namespace fapb {

// One part of the plan.  Its vertices are renumbered: 0..b-1 the boundary
// vertices in their local order, b..s-1 the inner ones by level, last
// eliminated first, so that N+(v) holds smaller numbers only.  All offsets
// are into the plan's arrays.
struct ElimPart {
  int32_t s, b;
  int32_t voff;        // loc / inv: s entries; eptr: s + 1 entries at voff + index of the part
  int32_t eptr_off;
  int32_t ent_off;     // ecol / eend / w0: nent entries, vertex after vertex
  int32_t nent;
  int32_t lev_off;     // nlev + 1 level starts, first level = highest (next to the boundary)
  int32_t nlev;
  int32_t boff;        // first boundary index of the part
  int32_t glev_off;    // gnlev + 1 level starts in units
  int32_t gnlev;
  int32_t stream_off;  // of the streams, in 16-byte words
  int32_t chunk_off, nchunks;
  int32_t nslots, sloc_off;
};

// Separator groups of the merge.  Rows eliminated one after the other are
// gathered while that costs no more: a group G shares the list U = N+ of its
// last vertex, which separates all of G from the rest, so with the parts'
// closed distances F
//   D[v][x] = min over u in U of F[v][u] + D[u][x]    for every v in G
// and the rows of a group are independent of one another: about ten levels
// instead of a hundred on grid parts, and every row u read serves four rows.
// Only boundary rows and rows that a list names (slots: boundary vertices
// first) stay in shared memory; the others, about two thirds on grid parts, go
// to memory straight from registers.  A unit is up to eight rows of a group;
// its list (slots) is padded to a multiple of four by repeating its last entry.
//
// The merge reads a part's units as a stream of chunks (consecutive units of
// one level, about kElimChunk16 * 16 bytes): the units' heads (body's offset in
// the chunk in 16-byte words, nu), then their bodies (rows, list as byte
// offsets into the strip, coefficients; elim_body16 words).  launch_elim_coef writes the stream.
struct ElimUnit {
  int32_t rows;   // first of kElimUnitRows rows: slot or -1, local index or -1
  int32_t list;   // first list entry
  int32_t nu;     // list entries, a multiple of four; kElimWide: eight rows, else at most four
  int32_t head;   // of the stream, in 8-byte words
  int32_t body;   // of the stream, in 16-byte words
  int32_t chunk;  // start of its chunk in the stream, in 16-byte words
};
struct ElimChunk {
  int32_t off, n16, nunits, pad_;  // in 16-byte words
};
// (18 KB: a barrier ends every chunk, and one of 8 KB held as few as two units of
// a grid part's first levels for 12 warps; merge of a 256 x 256 grid 12.8 ms at
// 8 KB, 9.8 at 18; two buffers of more would leave one CTA on an SM)
constexpr int32_t kElimChunk16 = 1152;
constexpr int32_t kElimWide = 1 << 30;
constexpr int kElimUnitRows = 8;
__host__ __device__ inline int32_t elim_body16(int32_t nu) {
  const int32_t k = nu & ~kElimWide;
  return kElimUnitRows / 2 + k / 4 + k * (nu & kElimWide ? 2 : 1);
}

// Array of a plan, not cleared when it is made: the parts' pieces are copied in
// by several threads, which then also take the page faults.
template <typename T>
struct PlanArray {
  std::unique_ptr<T[]> p;
  size_t n = 0;
  void make(size_t count) {
    p.reset(new T[count]);
    n = count;
  }
  T *data() { return p.get(); }
  const T *data() const { return p.get(); }
  size_t size() const { return n; }
  T &operator[](size_t i) { return p[i]; }
  const T &operator[](size_t i) const { return p[i]; }
};

struct ElimPlan {
  bool ok = false;
  std::vector<ElimPart> parts;
  PlanArray<int32_t> loc, inv;   // plan number <-> local index
  PlanArray<int32_t> eptr;       // entries of a vertex, relative to ent_off
  PlanArray<int32_t> ecol;       // N+(v), plan numbers, descending
  PlanArray<int32_t> eend;       // end of the entry's vertex, relative to ent_off
  PlanArray<int32_t> w0, w0b;    // weight (bits) of the arc v -> u, of u -> v (directed plans), or the sentinel
  PlanArray<int32_t> lev;
  PlanArray<ElimUnit> units;
  PlanArray<int32_t> glev, rows8;  // rows8: pairs (slot, local index)
  PlanArray<uint16_t> list;
  PlanArray<int32_t> sloc;  // local index of every slot, parts one after the other (sloc_off)
  PlanArray<ElimChunk> chunks;
  int64_t stream16 = 0;
  int32_t max_chunk16 = 0, max_chunks = 0;
  std::vector<int64_t> group_work;  // per part: list entries times padded rows
  int32_t max_s = 0, max_nent = 0, max_nlev = 0;
  int64_t nent = 0;
};

// Arcs of part p (0-based) for the plan: heads (local indices) and weights
// (bits), no self loops; of two arcs joining the same pair the later one counts.
struct ElimGraph {
  int32_t s = 0, b = 0, boff = 0;
  std::vector<int32_t> ptr, adj, w;  // w empty: weights come from a dense matrix
};

// Symbolic elimination of the parts on up to `threads` host threads; graph(p)
// fills in part p's adjacency and is called on any of them.  ok
// stays false when a part has more than kElimMaxS vertices (a strip of eight
// columns fills the shared memory) or more than s * max(s, 256) / kElimDense entries.
constexpr int32_t kElimMaxS = 6144;
constexpr int64_t kElimDense = 16;
// inf: bits of the sentinel; directed: keep both weights of an entry; groups:
// also build the separator groups.
void elim_build(int nparts, const std::function<void(int, ElimGraph *)> &graph, int threads, int32_t inf,
                bool directed, bool groups, ElimPlan *out);
// w0 of a one-part plan := offsets of the entries in a matrix whose rows and
// columns are the part's local indices.
void elim_offsets(int64_t ld, ElimPlan *plan);

// Device arrays of a plan.
struct ElimDev {
  const ElimPart *parts;
  const int32_t *loc, *inv, *eptr, *ecol, *eend, *w0, *w0b, *lev;
  const ElimUnit *units;
  const int32_t *glev, *rows8, *sloc;
  const uint16_t *list;
  const ElimChunk *chunks;
  int2 *ent;      // {plan number of u, W(v, u)}, written by launch_elim_up
  int32_t *entb;  // W(u, v); null: symmetric
  int32_t nparts, max_s, max_nent, max_nlev, max_chunk16, max_chunks;
};

// M (ld): the sentinel on nfill x nfill, 0 on the first nb diagonal entries,
// and the least weight of each listed arc (i, j, weight).
cudaError_t launch_elim_seed(int32_t *M, int64_t ld, int nb, int nfill, const int32_t *arcs, int narcs, cudaStream_t stream,
                             int64_t *launches);

// W of the listed parts (0-based plan parts; null: every part), and into M
// (boundary indices, symmetric parts only; null: not wanted) the shortest
// paths between a part's boundary vertices through its inner ones.  from: the
// edges' weights are the elements of this matrix that w0 names (offsets,
// elim_offsets) instead of w0 itself.
template <typename T>
cudaError_t launch_elim_up(const ElimDev &e, const int32_t *list, int count, const T *from, T *M, int64_t ldM,
                           cudaStream_t stream, int64_t *launches);

// Exact closures of the listed parts (as above) into out_off[i] + local row *
// ld + local column, from the exact distances of their boundary vertices: the
// closed boundary matrix dB (null with no rows: the parts have no boundary), or
// with `parts` (the listed parts' descriptors) the boundary rows of D, which
// hold every column (sorted position -> column: vid).
template <typename T>
struct ElimBoundary {
  const T *dB;
  int64_t ldB;
  const PartDesc *parts;
  const T *D;
  int64_t ldD;
  const int32_t *vid;
};
template <typename T>
cudaError_t launch_elim_close(const ElimDev &e, const int32_t *list, const int64_t *out_off, int count, int max_s,
                              const ElimBoundary<T> &bd, T *out, int64_t ld, cudaStream_t stream,
                              int64_t *launches);

// Rows of D for the listed boundary vertices (pairs boundary index, row of
// D), every column, from the closed dB; vid: sorted position -> column.
cudaError_t launch_elim_expand(const ElimDev &e, const int64_t *rows, int nrows, const int32_t *dB, int64_t ldB,
                               const int32_t *vid, int n, int32_t *D, int64_t ldD, cudaStream_t stream,
                               int64_t *launches);

// The listed parts' (pairs plan part, batch index of its PartDesc) streams:
// coefficients F[v][u] as int32 in s32 and, clamped at kMergeCap with both
// halves equal, in s16; maxA[plan part] = the largest finite distance from an
// inner to a boundary vertex.
constexpr int32_t kMergeCap = 32767;  // twice fits in 16 unsigned bits
struct ElimMerge {
  const int2 *list;
  int32_t count;
  int4 *s32, *s16;
  int32_t *maxA;
  unsigned long long *tiles;  // [2] strips run packed, strips run; null: int32 only
};
cudaError_t launch_elim_coef(const ElimDev &e, const ElimMerge &m, const PartDesc *parts, const int32_t *F,
                             int max_units, cudaStream_t stream, int64_t *launches);

// Inner rows of the listed parts' blocks from their boundary rows in D
// (stage 3); own columns from F.
cudaError_t launch_elim_merge(const ElimDev &e, const ElimMerge &m, const PartDesc *parts, const int32_t *F, int n,
                              int32_t *D, int64_t ldD, const int32_t *graph_id, const int32_t *ed2st, int max_slots,
                              cudaStream_t stream, int64_t *launches);
// Whether the numeric elimination of every part keeps its entries in a CTA's
// shared memory.
bool elim_up_fits(const ElimPlan &p, bool directed);
// CTAs of the merge that an SM holds for a part with that many slots (0 to 2).
int elim_merge_ctas(const ElimPlan &p, int slots);

}  // namespace fapb
