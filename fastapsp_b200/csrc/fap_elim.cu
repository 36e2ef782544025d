// Kernels of the vertex elimination (fap_elim.h): numeric elimination,
// closures and boundary rows by level-ordered sweeps over column strips held
// in shared memory.
#include "fap_elim.h"

#include <algorithm>
#include <type_traits>

#include "fap_common.cuh"

namespace fapb {
namespace {

constexpr int32_t kInf = FAP_INF_I32;
constexpr int kElimUpThreads = 1024;
constexpr int kUpLanes = 8;  // (lists hold 1 to 20 entries on road, geometric and grid parts)
constexpr int kElimSweepThreads = 512;
constexpr size_t kElimSmem = 226 * 1024;  // dynamic shared memory a CTA may take

// Strips of CW columns: row v of a strip starts at v * (CW + 1) words, so a
// row (lanes = columns) and a column (lanes = rows) are both conflict-free.
template <int CW>
constexpr int kStripLd = CW + 1;

__global__ void elim_seed_fill_kernel(int32_t *M, int64_t ld, int nb, int nfill) {
  const int64_t cols = (nfill + 3) / 4;
  const int64_t total = cols * nfill;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / cols, j = (t % cols) * 4;
    int4 x = make_int4(kInf, kInf, kInf, kInf);
    if (i < nb) {
      if (i == j) x.x = 0;
      if (i == j + 1) x.y = 0;
      if (i == j + 2) x.z = 0;
      if (i == j + 3) x.w = 0;
    }
    *reinterpret_cast<int4 *>(M + i * ld + j) = x;
  }
}

__global__ void elim_seed_arcs_kernel(int32_t *M, int64_t ld, const int32_t *__restrict__ arcs, int narcs) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= narcs) return;
  atomicMin(M + (int64_t)arcs[3 * t] * ld + arcs[3 * t + 1], arcs[3 * t + 2]);
}

// Numeric elimination, one CTA per part, levels from the first eliminated
// on; kUpLanes lanes take one entry (v, u_i), each some of v's later entries
// u_j: the entry (u_i, u_j), found in u_i's list, is lowered to
// W(v, u_i) + W(v, u_j).  Two vertices of a level may lower the same entry
// (atomicMin); none of them reads it before the level's barrier.
// Bound by the latency of the levels, so shared memory holds all that a level
// reads (ALL): entries as {u | entries after this one << 16, W}, the lists'
// starts and the levels' entry ranges (a 670-vertex boundary graph: 140 us
// with only W there, 58 us).  Parts of up to 38,000 entries (23,000 directed)
// whose whole plan does not fit keep W and u there, which the updates and the
// searches touch, and read starts and ends through L1.  (With the entries in L2
// larger parts took longer than their Floyd-Warshall; they keep that.)
// Directed parts (entb): an entry carries both weights, and a pair lowers both.
template <typename T, bool ALL>
__global__ void __launch_bounds__(kElimUpThreads)
    elim_up_kernel(ElimDev e, const int32_t *__restrict__ list, const T *__restrict__ from, T *M, int64_t ldM) {
  extern __shared__ int2 up_smem[];
  const ElimPart P = e.parts[list ? list[blockIdx.x] : blockIdx.x];
  const int32_t *eptr = e.eptr + P.eptr_off, *lev = e.lev + P.lev_off;
  const int32_t *ecol = e.ecol + P.ent_off, *eend = e.eend + P.ent_off, *w0 = e.w0 + P.ent_off;
  const T inf = Dist<T>::inf();
  const bool directed = e.entb != nullptr;
  int2 *gent = e.ent + P.ent_off;
  int32_t *gentb = directed ? e.entb + P.ent_off : nullptr;
  // ALL: entries, s + 1 list starts, nlev + 1 entry ranges, second weights;
  // else weights, second weights, heads
  int2 *ent = up_smem;
  int32_t *sptr = reinterpret_cast<int32_t *>(up_smem + P.nent), *slev = sptr + P.s + 1;
  int32_t *sw = reinterpret_cast<int32_t *>(up_smem);
  int32_t *entb = ALL ? slev + P.nlev + 1 : sw + P.nent;
  uint16_t *su = reinterpret_cast<uint16_t *>(entb + (directed ? P.nent : 0));
  const int lane = threadIdx.x % kUpLanes, group = threadIdx.x / kUpLanes, ngroups = blockDim.x / kUpLanes;
  auto value = [](int32_t bits) -> T {
    if constexpr (std::is_same<T, float>::value) return __int_as_float(bits);
    else return bits;
  };
  auto bits = [](T x) -> int32_t {
    if constexpr (std::is_same<T, float>::value) return __float_as_int(x);
    else return x;
  };
  auto entry = [&](int i) -> int2 {  // {head, W}
    if (ALL) return make_int2(ent[i].x & 0xffff, ent[i].y);
    return make_int2(su[i], sw[i]);
  };
  if (ALL) {
    for (int v = threadIdx.x; v <= P.s; v += blockDim.x) sptr[v] = eptr[v];
    for (int l = threadIdx.x; l <= P.nlev; l += blockDim.x) slev[l] = eptr[lev[l]];
  }
  for (int i = threadIdx.x; i < P.nent; i += blockDim.x) {
    const int32_t w = from ? bits(from[w0[i]]) : w0[i];
    if (ALL) {
      ent[i] = make_int2(ecol[i] | (eend[i] - i - 1) << 16, w);
    } else {
      sw[i] = w;
      su[i] = (uint16_t)ecol[i];
    }
    if (directed) entb[i] = e.w0b[P.ent_off + i];
  }
  __syncthreads();
  for (int l = P.nlev - 1; l >= 0; l--) {
    const int i1 = ALL ? slev[l + 1] : __ldg(eptr + __ldg(lev + l + 1));
    for (int i = (ALL ? slev[l] : __ldg(eptr + __ldg(lev + l))) + group; i < i1; i += ngroups) {
      const int end = ALL ? i + 1 + (int)((uint32_t)ent[i].x >> 16) : __ldg(eend + i);
      const int2 a = entry(i);
      const int ui = a.x;
      if (ui < P.b && M == nullptr) continue;  // (pairs of boundary vertices are not wanted)
      const T out = value(a.y), in = directed ? value(entb[i]) : out;
      if (out >= inf && in >= inf) continue;
      int lo = 0, hi = 0;
      if (ui >= P.b) {
        lo = ALL ? sptr[ui] : __ldg(eptr + ui);
        hi = ALL ? sptr[ui + 1] : __ldg(eptr + ui + 1);
      }
      for (int j = i + 1 + lane; j < end; j += kUpLanes) {
        const int2 c = entry(j);
        const int uj = c.x;
        const T fwd = in + value(c.y);  // u_i -> v -> u_j
        const T back = directed ? value(entb[j]) + out : fwd;
        if (fwd >= inf && back >= inf) continue;
        if (ui < P.b) {
          Dist<T>::atomic_min(M + (int64_t)(P.boff + ui) * ldM + P.boff + uj, fwd);
          Dist<T>::atomic_min(M + (int64_t)(P.boff + uj) * ldM + P.boff + ui, fwd);
          continue;
        }
        int x = lo, y = hi - 1;  // descending; u_j is in the list
        while (x < y) {
          const int m = (x + y) >> 1;
          if ((ALL ? ent[m].x & 0xffff : (int)su[m]) > uj) x = m + 1;
          else y = m;
        }
        // (non-negative float bits order like int32)
        if (fwd < inf) atomicMin(ALL ? &ent[x].y : sw + x, bits(fwd));
        if (directed && back < inf) atomicMin(entb + x, bits(back));
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < P.nent; i += blockDim.x) {
    gent[i] = entry(i);
    if (directed) gentb[i] = entb[i];
  }
}

// What a sweep reads of a part's plan: the entries, the lists' starts and the
// levels, in shared memory behind the strip (SM) or in global memory.
struct SweepPlan {
  const int2 *ent;
  const int32_t *entb;
  const int32_t *eptr, *lev;
};
template <int CW, bool SM>
__device__ __forceinline__ SweepPlan stage_plan(const ElimDev &e, const ElimPart &P, void *strip) {
  SweepPlan p{e.ent + P.ent_off, e.entb ? e.entb + P.ent_off : nullptr, e.eptr + P.eptr_off, e.lev + P.lev_off};
  if (!SM) return p;
  int2 *ent = reinterpret_cast<int2 *>(static_cast<int32_t *>(strip) + ((P.s * kStripLd<CW> + 1) & ~1));
  int32_t *eptr = reinterpret_cast<int32_t *>(ent + P.nent), *lev = eptr + P.s + 1, *entb = lev + P.nlev + 1;
  for (int i = threadIdx.x; i < P.nent; i += blockDim.x) ent[i] = __ldg(p.ent + i);
  for (int i = threadIdx.x; i <= P.s; i += blockDim.x) eptr[i] = __ldg(p.eptr + i);
  for (int i = threadIdx.x; i <= P.nlev; i += blockDim.x) lev[i] = __ldg(p.lev + i);
  if (p.entb)
    for (int i = threadIdx.x; i < P.nent; i += blockDim.x) entb[i] = __ldg(p.entb + i);
  return SweepPlan{ent, p.entb ? entb : nullptr, eptr, lev};
}
template <int CW>
size_t sweep_bytes(const ElimDev &e, int max_s, bool plan) {
  size_t words = ((size_t)max_s * kStripLd<CW> + 1) & ~size_t(1);
  if (plan) words += (e.entb ? 3 : 2) * (size_t)e.max_nent + (size_t)max_s + 1 + e.max_nlev + 1;
  return words * sizeof(int32_t);
}
template <typename T>
__device__ __forceinline__ T weight_of(int32_t bits) {
  if constexpr (std::is_same<T, float>::value) return __int_as_float(bits);
  else return bits;
}

// Rows of the inner vertices, level by level away from the boundary.  The
// first levels of a grid part hold one to three vertices with up to 200
// entries each: a level narrower than the CTA's row groups splits every list
// over several of them, which lower the row with atomic minima (nothing else
// reads it before the level's barrier; 16 closures of a 128 x 128 grid's
// parts: 1.46 ms without, 0.69 ms with).  Parts with short lists (at most 8
// entries on average) take whole lists: road114k 0.42 ms without the split,
// 0.52 with it.
template <typename T, int CW>
__device__ __forceinline__ void sweep_down(T *st, const ElimPart &P, const SweepPlan &p) {
  static_assert(32 % CW == 0, "a warp holds whole rows");
  const int c = threadIdx.x % CW, first = threadIdx.x / CW, step = blockDim.x / CW;
  const bool split = P.nent > 8 * (P.s - P.b);
  for (int l = 0; l < P.nlev; l++) {
    const int v0 = p.lev[l], v1 = p.lev[l + 1];
    const int sh = split ? 31 - __clz(max(step / (v1 - v0), 1)) : 0;  // (no level is empty)
    if (sh == 0) {
      for (int v = v0 + first; v < v1; v += step) {
        T *q = st + v * kStripLd<CW> + c;
        T acc = *q;
        const int e1 = p.eptr[v + 1];
#pragma unroll 4
        for (int i = p.eptr[v]; i < e1; i++) {
          const int2 x = p.ent[i];
          acc = Dist<T>::relax(weight_of<T>(x.y), st[x.x * kStripLd<CW> + c], acc);
        }
        *q = acc;
      }
    } else if (const int v = v0 + (first >> sh); v < v1) {
      T acc = Dist<T>::inf();
      const int e1 = p.eptr[v + 1];
#pragma unroll 2
      for (int i = p.eptr[v] + (first & ((1 << sh) - 1)); i < e1; i += 1 << sh) {
        const int2 x = p.ent[i];
        acc = Dist<T>::relax(weight_of<T>(x.y), st[x.x * kStripLd<CW> + c], acc);
      }
      if (acc < Dist<T>::inf()) Dist<T>::atomic_min(st + v * kStripLd<CW> + c, acc);
    }
    __syncthreads();
  }
}

// Exact closures.  CTA (strip, part): columns x0 .. x0 + CW - 1 (local
// indices) of the part's closed matrix.  Forward: y[v] = shortest path from v
// to the column's vertex x through vertices eliminated before v; only the
// vertices that x's first N+ entries lead to, one after the other, have one,
// so one warp walks them per column, without barriers.  Boundary: z = dB (x) y
// over the part's boundary vertices; a row read after another warp lowered it
// holds a path length between y and z, so the minimum is the same.  Backward:
// the remaining rows, level by level.  Bound by the latency of the walk and
// of the levels (road parts: ~50 of each): the plan sits in shared memory
// when three CTAs still fit on an SM with it (road114k: 827 us with a level
// barrier in the forward sweep and the plan in L1, 428 us).
// Boundary rows given in D (parts != null) are taken as they are.
template <typename T, int CW, bool SM>
__global__ void __launch_bounds__(kElimSweepThreads)
    elim_close_kernel(ElimDev e, const int32_t *__restrict__ list, const int64_t *__restrict__ out_off,
                      ElimBoundary<T> bd, T *out, int64_t ld) {
  extern __shared__ __align__(16) int32_t close_smem[];
  T *st = reinterpret_cast<T *>(close_smem);
  const T inf = Dist<T>::inf();
  const ElimPart P = e.parts[list ? list[blockIdx.y] : blockIdx.y];
  const int x0 = blockIdx.x * CW;
  if (x0 >= P.s) return;
  const int nx = min(CW, P.s - x0);
  const int32_t *loc = e.loc + P.voff, *inv = e.inv + P.voff;
  const int c = threadIdx.x % CW, first = threadIdx.x / CW, step = blockDim.x / CW;
  const int lane = threadIdx.x & 31;
  const SweepPlan p = stage_plan<CW, SM>(e, P, st);
  for (int i = threadIdx.x; i < P.s * kStripLd<CW>; i += blockDim.x) st[i] = inf;
  __syncthreads();
  for (int x = threadIdx.x >> 5; x < nx; x += blockDim.x >> 5) {
    int v = inv[x0 + x];
    if (lane == 0) st[v * kStripLd<CW> + x] = T(0);
    __syncwarp();
    while (v >= P.b) {
      const int e0 = p.eptr[v], e1 = p.eptr[v + 1];
      if (e0 == e1) break;
      const T y = st[v * kStripLd<CW> + x];
      const int up = p.ent[e0].x;
      if (y < inf)
        for (int i = e0 + lane; i < e1; i += 32) {
          const int2 a = p.ent[i];
          T *q = st + a.x * kStripLd<CW> + x;
          *q = Dist<T>::relax(weight_of<T>(p.entb ? p.entb[i] : a.y), y, *q);
        }
      __syncwarp();
      v = up;
    }
  }
  __syncthreads();
  if (bd.parts != nullptr) {
    const PartDesc pd = bd.parts[blockIdx.y];
    const T *D = bd.D + pd.row_base * bd.ldD + (c < nx ? __ldg(bd.vid + pd.start + x0 + c) : 0);
    for (int k = first; k < P.b; k += step) st[k * kStripLd<CW> + c] = D[k * bd.ldD];
    __syncthreads();
  } else if (P.b > 0) {
    for (int k = first; k < P.b; k += step) {
      const T *row = bd.dB + (int64_t)(P.boff + k) * bd.ldB + P.boff;
      T acc = st[k * kStripLd<CW> + c];
#pragma unroll 4
      for (int q = 0; q < P.b; q++) acc = Dist<T>::relax(__ldg(row + q), st[q * kStripLd<CW> + c], acc);
      st[k * kStripLd<CW> + c] = acc;
    }
    __syncthreads();
  }
  sweep_down<T, CW>(st, P, p);
  if (c < nx) {
    T *o = out + out_off[blockIdx.y] + x0 + c;
    for (int v = first; v < P.s; v += step) o[loc[v] * ld] = st[v * kStripLd<CW> + c];
  }
}

// Boundary rows of D.  CTA (strip of CW listed boundary vertices g, part q):
// D[g][v] for q's vertices v, from dB[g][.] at q's boundary vertices (the
// distances are symmetric, so the strip's columns are the g); stored row by
// row at q's columns.
template <int CW, bool SM>
__global__ void __launch_bounds__(kElimSweepThreads)
    elim_expand_kernel(ElimDev e, const int64_t *__restrict__ rows, int nrows, const int32_t *__restrict__ dB,
                       int64_t ldB, const int32_t *__restrict__ vid, int n, int32_t *D, int64_t ldD) {
  extern __shared__ __align__(16) int32_t st[];
  const ElimPart P = e.parts[blockIdx.y];
  const int r0 = blockIdx.x * CW, nr = min(CW, nrows - r0);
  const SweepPlan p = stage_plan<CW, SM>(e, P, st);
  for (int i = threadIdx.x; i < P.s * kStripLd<CW>; i += blockDim.x) st[i] = kInf;
  __syncthreads();
  for (int i = threadIdx.x; i < nr * P.b; i += blockDim.x) {
    const int r = i / P.b, k = i - r * P.b;
    st[k * kStripLd<CW> + r] = __ldg(dB + rows[2 * (r0 + r)] * ldB + P.boff + k);
  }
  __syncthreads();
  sweep_down<int32_t, CW>(st, P, p);
  const int32_t *inv = e.inv + P.voff;
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < nr; r += blockDim.x >> 5) {
    int32_t *row = D + rows[2 * (r0 + r) + 1] * ldD;
    for (int i = lane; i < P.s; i += 32) row[vid[P.voff + i]] = st[inv[i] * kStripLd<CW> + r];
    if (blockIdx.y == 0)
      for (int64_t j = n + lane; j < ldD; j += 32) row[j] = kInf;
  }
}

// The groups' streams: a warp per unit, a lane per list entry.
__global__ void __launch_bounds__(256)
    elim_coef_kernel(ElimDev e, ElimMerge m, const PartDesc *__restrict__ parts, const int32_t *__restrict__ F) {
  const int2 w = m.list[blockIdx.y];
  const ElimPart P = e.parts[w.x];
  const PartDesc pd = parts[w.y];
  const int32_t *Fp = F + pd.f_off, *sloc = e.sloc + P.sloc_off;
  const int lane = threadIdx.x % 32;
  int4 *s32 = m.s32 + P.stream_off, *s16 = m.s16 + P.stream_off;
  int far = 0;
  const int u0 = e.glev[P.glev_off], u1 = e.glev[P.glev_off + P.gnlev];
  for (int i = u0 + (blockIdx.x * blockDim.x + threadIdx.x) / 32; i < u1; i += gridDim.x * blockDim.x / 32) {
    const ElimUnit U = e.units[i];
    const int nu = U.nu & ~kElimWide, chunks = U.nu & kElimWide ? 2 : 1;
    const int2 head = make_int2(U.body - U.chunk, U.nu);
    const int2 *rows = reinterpret_cast<const int2 *>(e.rows8) + U.rows;
    if (lane == 0) {
      reinterpret_cast<int2 *>(s32)[U.head] = head;
      reinterpret_cast<int2 *>(s16)[U.head] = head;
    }
    if (lane < kElimUnitRows) {
      reinterpret_cast<int2 *>(s32 + U.body)[lane] = rows[lane];
      reinterpret_cast<int2 *>(s16 + U.body)[lane] = rows[lane];
    }
    const int lists = U.body + kElimUnitRows / 2, coef = lists + nu / 4;
    for (int k = lane; k < nu; k += 32) {
      reinterpret_cast<int32_t *>(s32 + lists)[k] = e.list[U.list + k] * 128;
      reinterpret_cast<int32_t *>(s16 + lists)[k] = e.list[U.list + k] * 128;
    }
    for (int t = lane; t < nu * chunks; t += 32) {
      const int k = t / chunks, c = t - k * chunks;
      const int u = sloc[e.list[U.list + k]];
      int32_t x[4];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int v = rows[4 * c + r].y;
        x[r] = v < 0 ? kInf : __ldg(Fp + (int64_t)v * pd.ldf + u);
      }
      s32[coef + t] = make_int4(x[0], x[1], x[2], x[3]);
#pragma unroll
      for (int r = 0; r < 4; r++) x[r] = min(x[r], kMergeCap) * 0x10001;
      s16[coef + t] = make_int4(x[0], x[1], x[2], x[3]);
    }
  }
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < (P.s - P.b) * P.b; t += gridDim.x * blockDim.x) {
    const int32_t x = __ldg(Fp + (int64_t)(P.b + t / P.b) * pd.ldf + t % P.b);
    if (x < kInf) far = max(far, x);
  }
  far = __reduce_max_sync(0xffffffffu, far);
  if (lane == 0 && far > 0) atomicMax(m.maxA + w.x, far);
}

// How a strip sits in shared memory: kMergePacked, a lane's word is two
// columns in 16 unsigned bits (shifted by the column's offset and clamped at
// kMergeCap); kMergePair, a lane holds two columns as int32; kMergeOne, one.
enum MergeMode { kMergeOne, kMergePair, kMergePacked };

// Where a strip's rows go: the lane's column or columns of the block's rows in
// D, with the own-part columns taken from F (jx, jy: local index or -1).
struct MergeOut {
  char *D;       // first row, the lane's first column
  int32_t ld;    // bytes between rows
  const int32_t *F;
  int32_t ldf;
  int jx, jy, ox, oy;  // ox, oy: packed columns' offsets
};

// One unit of NR rows on a warp.  Per list entry one load of the strip serves
// NR rows; body: the unit's rows, list and coefficients in shared memory; st:
// the lane's place in row 0.  OWN: the strip has own-part columns; their values
// are asked for before the relaxations, which hide the latency.
template <int MODE, int NR, bool OWN>
__device__ __forceinline__ void merge_unit(char *st, const int4 *body, int nu, const MergeOut &o) {
  constexpr bool PK = MODE == kMergePacked, TWO = MODE == kMergePair;
  constexpr int LD = TWO ? 256 : 128;  // bytes of a strip's row; the lists are in units of 128
  const int4 *list = body + kElimUnitRows / 2, *coef = list + nu / 4;
  int acc[NR], acc2[TWO ? NR : 1], fx[OWN ? NR : 1], fy[OWN && MODE != kMergeOne ? NR : 1];
  if (OWN) {
#pragma unroll
    for (int r = 0; r < NR; r++) {
      const int v = max(reinterpret_cast<const int2 *>(body)[r].y, 0);
      const int32_t *f = o.F + (int64_t)v * o.ldf;
      if (o.jx >= 0) fx[r] = __ldg(f + o.jx);
      if (MODE != kMergeOne && o.jy >= 0) fy[MODE != kMergeOne ? r : 0] = __ldg(f + o.jy);
    }
  }
#pragma unroll
  for (int r = 0; r < NR; r++) {
    acc[r] = PK ? kMergeCap * 0x10001 : kInf;
    if (TWO) acc2[TWO ? r : 0] = kInf;
  }
  auto relax = [](int x, int y, int z) -> int {
    if (PK) return (int)__viaddmin_u16x2((unsigned)x, (unsigned)y, (unsigned)z);
    return __viaddmin_s32(x, y, z);
  };
  auto step = [&](int u, const int4 *f) {
    int x, y = 0;
    if (TWO) {
      const int2 t = *reinterpret_cast<const int2 *>(st + 2 * u);
      x = t.x;
      y = t.y;
    } else {
      x = *reinterpret_cast<const int *>(st + u);
    }
#pragma unroll
    for (int g = 0; g < NR / 4; g++) {
      const int4 a = f[g];
      const int c[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int r = 0; r < 4; r++) {
        acc[4 * g + r] = relax(c[r], x, acc[4 * g + r]);
        if (TWO) acc2[TWO ? 4 * g + r : 0] = relax(c[r], y, acc2[TWO ? 4 * g + r : 0]);
      }
    }
  };
#pragma unroll 2
  for (const int4 *end = coef; list < end; list++, coef += NR) {
    const int4 u = *list;
    step(u.x, coef);
    step(u.y, coef + NR / 4);
    step(u.z, coef + 2 * (NR / 4));
    step(u.w, coef + 3 * (NR / 4));
  }
#pragma unroll
  for (int r = 0; r < NR; r++) {
    const int2 v = reinterpret_cast<const int2 *>(body)[r];
    if (v.y < 0) break;
    int2 d = make_int2(acc[r], acc2[TWO ? r : 0]);
    if (v.x >= 0) {
      if (TWO) *reinterpret_cast<int2 *>(st + v.x * LD) = d;
      else *reinterpret_cast<int *>(st + v.x * LD) = d.x;
    }
    if (PK) {
      const int x = acc[r] & 0xffff, y = (int)((uint32_t)acc[r] >> 16);
      d = make_int2(__viaddmin_s32(x, o.ox, kInf), __viaddmin_s32(y, o.oy, kInf));
      if (x >= kMergeCap) d.x = kInf;
      if (y >= kMergeCap) d.y = kInf;
    }
    if (OWN && o.jx >= 0) d.x = fx[r];
    if (OWN && MODE != kMergeOne && o.jy >= 0) d.y = fy[MODE != kMergeOne ? r : 0];
    char *row = o.D + (int64_t)v.y * o.ld;
    if (MODE == kMergeOne) __stcs(reinterpret_cast<int *>(row), d.x);
    else __stcs(reinterpret_cast<int2 *>(row), d);
  }
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The part's chunks through a ring of kMergeRing buffers in shared memory,
// copied asynchronously a chunk ahead; a chunk's units are independent, a
// barrier ends every chunk.
constexpr int kMergeRing = 2;
template <int MODE, bool OWN>
__device__ __forceinline__ void merge_stream(char *st, int4 *ring, int buf16, const ElimChunk *chunks, int nchunks,
                                             const int4 *__restrict__ stream, const MergeOut &o) {
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  auto fetch = [&](int c) {
    if (c < nchunks) {
      const ElimChunk k = chunks[c];
      for (int i = threadIdx.x; i < k.n16; i += blockDim.x) cp_async16(ring + (c % kMergeRing) * buf16 + i, stream + k.off + i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  for (int c = 0; c < nchunks; c++) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // chunk c is here, and every warp is done with chunk c - 1
    fetch(c + 1);
    const int4 *buf = ring + (c % kMergeRing) * buf16;
    const int n = chunks[c].nunits;
    for (int i = warp; i < n; i += nwarps) {
      const int2 head = reinterpret_cast<const int2 *>(buf)[i];
      if (head.y & kElimWide) merge_unit<MODE, 8, OWN>(st, buf + head.x, head.y & ~kElimWide, o);
      else merge_unit<MODE, 4, OWN>(st, buf + head.x, head.y, o);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

constexpr int kMergeThreads = 384;
constexpr int kMergeCols = 64;
__host__ __device__ inline size_t merge_smem(int slots, int slot_bytes, int chunk16, int chunks) {
  return (size_t)slots * slot_bytes + ((size_t)kMergeRing * chunk16 + chunks) * 16;
}

// Inner rows.  CTA (strip of 64 columns, listed part).  The boundary rows of
// the strip give every column its least finite entry (off) and the strip its
// range; the rows are relaxed in packed 16 bits where maxA + range < kMergeCap
// (every inner row's shifted value is at most that sum, two values of at most
// kMergeCap do not overflow, and one at kMergeCap means no path), else in
// int32: two columns a lane (pair) where two CTAs still fit on an SM, else as
// two strips of 32 columns.  A grid part's row takes 28 relaxations (its
// boundary: 164), a geometric graph's 5 (27).  Bound by issue: about 100
// instructions per packed row of 64 columns, of which 39 relax.  Merge of a
// 256 x 256 grid 22.4 -> 9.8 ms, of a 60,000-vertex geometric graph 9.3 -> 5.5
// (the min-plus tiles before); 384 threads of 85 registers, since at 56 the
// pair form spills (9.7 ms).
__global__ void __launch_bounds__(kMergeThreads, 2)
    elim_merge_kernel(ElimDev e, ElimMerge m, const PartDesc *__restrict__ parts, const int32_t *__restrict__ F,
                      int n, int32_t *D, int64_t ldD, const int32_t *__restrict__ graph_id,
                      const int32_t *__restrict__ ed2st, int max_slots, int pair) {
  extern __shared__ __align__(16) int32_t st[];
  __shared__ int32_t lo[kMergeCols], hi[kMergeCols], own[kMergeCols];
  __shared__ int range, any_own;
  int4 *ring = reinterpret_cast<int4 *>(st + (size_t)max_slots * (pair ? 64 : 32));
  ElimChunk *chunks = reinterpret_cast<ElimChunk *>(ring + (size_t)kMergeRing * e.max_chunk16);
  const int2 w = m.list[blockIdx.y];
  const ElimPart P = e.parts[w.x];
  const PartDesc pd = parts[w.y];
  const int64_t c0 = (int64_t)blockIdx.x * kMergeCols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int32_t *Dp = D + pd.row_base * ldD + c0;
  for (int i = threadIdx.x; i < P.nchunks; i += blockDim.x) chunks[i] = e.chunks[P.chunk_off + i];
  if (threadIdx.x == 0) range = any_own = 0;
  if (threadIdx.x < kMergeCols) {
    lo[threadIdx.x] = kInf;
    hi[threadIdx.x] = 0;
  }
  __syncthreads();
  if (threadIdx.x < kMergeCols) {
    const int64_t v = c0 + threadIdx.x;
    int j = -1;
    if (v < n && __ldg(graph_id + v) == pd.part) {
      j = __ldg(ed2st + v) - pd.start;
      any_own = 1;
    }
    own[threadIdx.x] = j;
  }
  if (m.tiles != nullptr) {
    int mn[2] = {kInf, kInf}, mx[2] = {0, 0};
#pragma unroll 4
    for (int k = warp; k < P.b; k += nwarps) {
      const int2 x = reinterpret_cast<const int2 *>(Dp + (int64_t)k * ldD)[lane];
      mn[0] = min(mn[0], x.x);
      mn[1] = min(mn[1], x.y);
      if (x.x < kInf) mx[0] = max(mx[0], x.x);
      if (x.y < kInf) mx[1] = max(mx[1], x.y);
    }
#pragma unroll
    for (int t = 0; t < 2; t++) {
      atomicMin(&lo[2 * lane + t], mn[t]);
      atomicMax(&hi[2 * lane + t], mx[t]);
    }
    __syncthreads();
    if (threadIdx.x < kMergeCols && lo[threadIdx.x] < kInf) atomicMax(&range, hi[threadIdx.x] - lo[threadIdx.x]);
  }
  __syncthreads();
  const bool pk = m.tiles != nullptr && range < kMergeCap && m.maxA[w.x] + range < kMergeCap;
  if (threadIdx.x == 0 && m.tiles != nullptr) {
    atomicAdd(m.tiles + 1, 1ull);
    if (pk) atomicAdd(m.tiles, 1ull);
  }
  MergeOut o{reinterpret_cast<char *>(Dp + 2 * lane), (int32_t)(ldD * 4), F + pd.f_off, pd.ldf, 0, 0, 0, 0};
  o.jx = own[2 * lane];
  o.jy = own[2 * lane + 1];
  char *lst = reinterpret_cast<char *>(st + lane);
  if (pk) {
    o.ox = lo[2 * lane];
    o.oy = lo[2 * lane + 1];
#pragma unroll 4
    for (int k = warp; k < P.b; k += nwarps) {
      const int2 x = reinterpret_cast<const int2 *>(Dp + (int64_t)k * ldD)[lane];
      const int a = x.x >= kInf ? kMergeCap : min(x.x - o.ox, kMergeCap);
      const int b = x.y >= kInf ? kMergeCap : min(x.y - o.oy, kMergeCap);
      st[k * 32 + lane] = a | b << 16;
    }
    if (any_own) merge_stream<kMergePacked, true>(lst, ring, e.max_chunk16, chunks, P.nchunks, m.s16 + P.stream_off, o);
    else merge_stream<kMergePacked, false>(lst, ring, e.max_chunk16, chunks, P.nchunks, m.s16 + P.stream_off, o);
    return;
  }
  if (pair) {
#pragma unroll 4
    for (int k = warp; k < P.b; k += nwarps)
      reinterpret_cast<int2 *>(st)[k * 32 + lane] = reinterpret_cast<const int2 *>(Dp + (int64_t)k * ldD)[lane];
    lst = reinterpret_cast<char *>(st + 2 * lane);
    if (any_own) merge_stream<kMergePair, true>(lst, ring, e.max_chunk16, chunks, P.nchunks, m.s32 + P.stream_off, o);
    else merge_stream<kMergePair, false>(lst, ring, e.max_chunk16, chunks, P.nchunks, m.s32 + P.stream_off, o);
    return;
  }
  for (int h = 0; h < 2; h++) {
#pragma unroll 4
    for (int k = warp; k < P.b; k += nwarps) st[k * 32 + lane] = Dp[(int64_t)k * ldD + 32 * h + lane];
    o.D = reinterpret_cast<char *>(Dp + 32 * h + lane);
    o.jx = own[32 * h + lane];
    if (any_own) merge_stream<kMergeOne, true>(lst, ring, e.max_chunk16, chunks, P.nchunks, m.s32 + P.stream_off, o);
    else merge_stream<kMergeOne, false>(lst, ring, e.max_chunk16, chunks, P.nchunks, m.s32 + P.stream_off, o);
  }
}

// Shared memory of elim_up_kernel<ALL>.
size_t up_smem_bytes(bool all, int32_t max_nent, int32_t max_s, int32_t max_nlev, bool directed) {
  const size_t n = max_nent;
  if (!all) return n * (directed ? 10 : 6);
  return (n * (directed ? 3 : 2) + (size_t)max_s + max_nlev + 2) * sizeof(int32_t);
}

template <class K>
cudaError_t allow_smem(K kern, size_t smem) {
  return smem > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                          : cudaSuccess;
}

// Strip width and whether the plan is staged: 8 columns with the plan (four
// CTAs on an SM for road parts; road114k's closures 0.42 ms, 0.55 ms with 16
// columns staged or not), then 16 without (grid parts, whose 20,000 entries
// leave no room: 0.68 ms against 0.81 with 8), then 8 without.
constexpr size_t kElimHalf = 113 * 1024;  // two CTAs on an SM
template <class F>
cudaError_t for_strip(const ElimDev &e, int max_s, F run) {
  using C16 = std::integral_constant<int, 16>;
  using C8 = std::integral_constant<int, 8>;
  if (sweep_bytes<8>(e, max_s, true) <= kElimHalf) return run(C8(), std::true_type());
  if (sweep_bytes<16>(e, max_s, false) <= kElimHalf) return run(C16(), std::false_type());
  return run(C8(), std::false_type());
}

}  // namespace

cudaError_t launch_elim_seed(int32_t *M, int64_t ld, int nb, int nfill, const int32_t *arcs, int narcs,
                             cudaStream_t stream, int64_t *launches) {
  if (nb <= 0) return cudaSuccess;
  if (ld % 4 != 0 || nfill < nb || nfill > ld) return cudaErrorInvalidValue;
  const int64_t total = ((int64_t)nfill + 3) / 4 * nfill;
  elim_seed_fill_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 4096), 256, 0, stream>>>(M, ld, nb, nfill);
  *launches += 1;
  if (narcs > 0) {
    elim_seed_arcs_kernel<<<(narcs + 255) / 256, 256, 0, stream>>>(M, ld, arcs, narcs);
    *launches += 1;
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_elim_up(const ElimDev &e, const int32_t *list, int count, const T *from, T *M, int64_t ldM,
                           cudaStream_t stream, int64_t *launches) {
  if (list == nullptr) count = e.nparts;
  if (count <= 0) return cudaSuccess;
  if (M != nullptr && e.entb != nullptr) return cudaErrorInvalidValue;
  const bool directed = e.entb != nullptr;
  const bool all = up_smem_bytes(true, e.max_nent, e.max_s, e.max_nlev, directed) <= kElimSmem;
  const size_t smem = up_smem_bytes(all, e.max_nent, e.max_s, e.max_nlev, directed);
  if (smem > kElimSmem) return cudaErrorInvalidValue;  // (elim_up_fits)
  auto kern = all ? elim_up_kernel<T, true> : elim_up_kernel<T, false>;
  cudaError_t err = allow_smem(kern, smem);
  if (err != cudaSuccess) return err;
  kern<<<count, kElimUpThreads, smem, stream>>>(e, list, from, M, ldM);
  *launches += 1;
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_elim_close(const ElimDev &e, const int32_t *list, const int64_t *out_off, int count, int max_s,
                              const ElimBoundary<T> &bd, T *out, int64_t ld, cudaStream_t stream,
                              int64_t *launches) {
  if (count <= 0 || max_s <= 0) return cudaSuccess;
  return for_strip(e, max_s, [&](auto cw, auto sm) -> cudaError_t {
    constexpr int CW = decltype(cw)::value;
    constexpr bool SM = decltype(sm)::value;
    const size_t smem = sweep_bytes<CW>(e, max_s, SM);
    cudaError_t err = allow_smem(elim_close_kernel<T, CW, SM>, smem);
    if (err != cudaSuccess) return err;
    elim_close_kernel<T, CW, SM><<<dim3((max_s + CW - 1) / CW, count), kElimSweepThreads, smem, stream>>>(
        e, list, out_off, bd, out, ld);
    *launches += 1;
    return cudaGetLastError();
  });
}

#define FAPB_ELIM(T)                                                                                             \
  template cudaError_t launch_elim_up<T>(const ElimDev &, const int32_t *, int, const T *, T *, int64_t,        \
                                         cudaStream_t, int64_t *);                                              \
  template cudaError_t launch_elim_close<T>(const ElimDev &, const int32_t *, const int64_t *, int, int,        \
                                            const ElimBoundary<T> &, T *, int64_t, cudaStream_t, int64_t *);
FAPB_ELIM(int32_t)
FAPB_ELIM(float)
#undef FAPB_ELIM

cudaError_t launch_elim_expand(const ElimDev &e, const int64_t *rows, int nrows, const int32_t *dB, int64_t ldB,
                               const int32_t *vid, int n, int32_t *D, int64_t ldD, cudaStream_t stream,
                               int64_t *launches) {
  if (nrows <= 0 || e.nparts <= 0) return cudaSuccess;
  return for_strip(e, e.max_s, [&](auto cw, auto sm) -> cudaError_t {
    constexpr int CW = decltype(cw)::value;
    constexpr bool SM = decltype(sm)::value;
    const size_t smem = sweep_bytes<CW>(e, e.max_s, SM);
    cudaError_t err = allow_smem(elim_expand_kernel<CW, SM>, smem);
    if (err != cudaSuccess) return err;
    elim_expand_kernel<CW, SM><<<dim3((nrows + CW - 1) / CW, e.nparts), kElimSweepThreads, smem, stream>>>(
        e, rows, nrows, dB, ldB, vid, n, D, ldD);
    *launches += 1;
    return cudaGetLastError();
  });
}

bool elim_up_fits(const ElimPlan &p, bool directed) {
  return up_smem_bytes(false, p.max_nent, p.max_s, p.max_nlev, directed) <= kElimSmem ||
         up_smem_bytes(true, p.max_nent, p.max_s, p.max_nlev, directed) <= kElimSmem;
}

int elim_merge_ctas(const ElimPlan &p, int slots) {
  const size_t smem = merge_smem(slots, 128, p.max_chunk16, p.max_chunks);
  return smem <= kElimHalf ? 2 : smem <= kElimSmem ? 1 : 0;
}

cudaError_t launch_elim_coef(const ElimDev &e, const ElimMerge &m, const PartDesc *parts, const int32_t *F,
                             int max_units, cudaStream_t stream, int64_t *launches) {
  if (m.count <= 0) return cudaSuccess;
  cudaError_t err = cudaMemsetAsync(m.maxA, 0, (size_t)e.nparts * sizeof(int32_t), stream);
  if (err != cudaSuccess) return err;
  elim_coef_kernel<<<dim3(std::max(1, std::min(16, (max_units + 7) / 8)), m.count), 256, 0, stream>>>(e, m, parts, F);
  *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_elim_merge(const ElimDev &e, const ElimMerge &m, const PartDesc *parts, const int32_t *F, int n,
                              int32_t *D, int64_t ldD, const int32_t *graph_id, const int32_t *ed2st, int max_slots,
                              cudaStream_t stream, int64_t *launches) {
  if (m.count <= 0) return cudaSuccess;
  if (ldD % kMergeCols != 0 || ldD > INT32_MAX / 4) return cudaErrorInvalidValue;
  const bool pair = merge_smem(max_slots, 256, e.max_chunk16, e.max_chunks) <= kElimHalf;
  const size_t smem = merge_smem(max_slots, pair ? 256 : 128, e.max_chunk16, e.max_chunks);
  if (smem > kElimSmem) return cudaErrorInvalidValue;
  cudaError_t err = allow_smem(elim_merge_kernel, smem);
  if (err != cudaSuccess) return err;
  elim_merge_kernel<<<dim3((unsigned)(ldD / kMergeCols), m.count), kMergeThreads, smem, stream>>>(
      e, m, parts, F, n, D, ldD, graph_id, ed2st, max_slots, pair ? 1 : 0);
  *launches += 1;
  return cudaGetLastError();
}

}  // namespace fapb
