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
// Bound by the latency of the levels, so SM keeps all that a level reads in
// shared memory: entries as {u | entries after this one << 16, W}, the lists'
// starts and the levels' entry ranges (a 670-vertex boundary graph: 140 us
// with only W there, 58 us).  Otherwise the entries sit in L2 and are read
// past L1.
template <bool SM>
__global__ void __launch_bounds__(kElimUpThreads)
    elim_up_kernel(ElimDev e, const int32_t *__restrict__ from, int32_t *M, int64_t ldM) {
  extern __shared__ int2 up_smem[];
  const ElimPart P = e.parts[blockIdx.x];
  const int32_t *eptr = e.eptr + P.eptr_off, *lev = e.lev + P.lev_off;
  const int32_t *ecol = e.ecol + P.ent_off, *eend = e.eend + P.ent_off, *w0 = e.w0 + P.ent_off;
  int2 *gent = e.ent + P.ent_off;
  int2 *ent = SM ? up_smem : gent;
  int32_t *sptr = reinterpret_cast<int32_t *>(up_smem + (SM ? P.nent : 0));  // s + 1 list starts
  int32_t *slev = sptr + P.s + 1;                                            // nlev + 1 entry ranges
  const int lane = threadIdx.x % kUpLanes, group = threadIdx.x / kUpLanes, ngroups = blockDim.x / kUpLanes;
  if (SM) {
    for (int v = threadIdx.x; v <= P.s; v += blockDim.x) sptr[v] = eptr[v];
    for (int l = threadIdx.x; l <= P.nlev; l += blockDim.x) slev[l] = eptr[lev[l]];
  }
  for (int i = threadIdx.x; i < P.nent; i += blockDim.x)
    ent[i] = make_int2(SM ? ecol[i] | (eend[i] - i - 1) << 16 : ecol[i], from ? from[w0[i]] : w0[i]);
  if (!SM) __threadfence();
  __syncthreads();
  for (int l = P.nlev - 1; l >= 0; l--) {
    const int i1 = SM ? slev[l + 1] : eptr[lev[l + 1]];
    for (int i = (SM ? slev[l] : eptr[lev[l]]) + group; i < i1; i += ngroups) {
      const int2 a = SM ? ent[i] : __ldcg(ent + i);
      const int ui = SM ? a.x & 0xffff : a.x;
      const int end = SM ? i + 1 + (int)((uint32_t)a.x >> 16) : eend[i];
      if (a.y >= kInf) continue;
      int lo = 0, hi = 0;
      if (ui >= P.b) {
        lo = SM ? sptr[ui] : eptr[ui];
        hi = SM ? sptr[ui + 1] : eptr[ui + 1];
      }
      for (int j = i + 1 + lane; j < end; j += kUpLanes) {
        const int2 c = SM ? ent[j] : __ldcg(ent + j);
        const int uj = SM ? c.x & 0xffff : c.x;
        const int32_t w = a.y + c.y;
        if (w >= kInf) continue;
        if (ui < P.b) {
          atomicMin(M + (int64_t)(P.boff + ui) * ldM + P.boff + uj, w);
          atomicMin(M + (int64_t)(P.boff + uj) * ldM + P.boff + ui, w);
          continue;
        }
        int x = lo, y = hi - 1;  // descending; u_j is in the list
        while (x < y) {
          const int m = (x + y) >> 1;
          if ((SM ? ent[m].x & 0xffff : ecol[m]) > uj) x = m + 1;
          else y = m;
        }
        atomicMin(&ent[x].y, w);
      }
    }
    __syncthreads();
  }
  if (SM)
    for (int i = threadIdx.x; i < P.nent; i += blockDim.x) gent[i] = make_int2(ent[i].x & 0xffff, ent[i].y);
}

// What a sweep reads of a part's plan: the entries, the lists' starts and the
// levels, in shared memory behind the strip (SM) or in global memory.
struct SweepPlan {
  const int2 *ent;
  const int32_t *eptr, *lev;
};
template <int CW, bool SM>
__device__ __forceinline__ SweepPlan stage_plan(const ElimDev &e, const ElimPart &P, int32_t *st) {
  SweepPlan p{e.ent + P.ent_off, e.eptr + P.eptr_off, e.lev + P.lev_off};
  if (!SM) return p;
  int2 *ent = reinterpret_cast<int2 *>(st + ((P.s * kStripLd<CW> + 1) & ~1));
  int32_t *eptr = reinterpret_cast<int32_t *>(ent + P.nent), *lev = eptr + P.s + 1;
  for (int i = threadIdx.x; i < P.nent; i += blockDim.x) ent[i] = __ldg(p.ent + i);
  for (int i = threadIdx.x; i <= P.s; i += blockDim.x) eptr[i] = __ldg(p.eptr + i);
  for (int i = threadIdx.x; i <= P.nlev; i += blockDim.x) lev[i] = __ldg(p.lev + i);
  return SweepPlan{ent, eptr, lev};
}
template <int CW>
size_t sweep_bytes(const ElimDev &e, int max_s, bool plan) {
  size_t words = ((size_t)max_s * kStripLd<CW> + 1) & ~size_t(1);
  if (plan) words += 2 * (size_t)e.max_nent + (size_t)max_s + 1 + e.max_nlev + 1;
  return words * sizeof(int32_t);
}

// Rows of the inner vertices, level by level away from the boundary.  The
// first levels of a grid part hold one to three vertices with up to 200
// entries each: a level narrower than the CTA's row groups splits every list
// over several of them, which lower the row with atomic minima (nothing else
// reads it before the level's barrier; 16 closures of a 128 x 128 grid's
// parts: 1.46 ms without, 0.69 ms with).  Parts with short lists (at most 8
// entries on average) take whole lists: road114k 0.42 ms without the split,
// 0.52 with it.
template <int CW>
__device__ __forceinline__ void sweep_down(int32_t *st, const ElimPart &P, const SweepPlan &p) {
  static_assert(32 % CW == 0, "a warp holds whole rows");
  const int c = threadIdx.x % CW, first = threadIdx.x / CW, step = blockDim.x / CW;
  const bool split = P.nent > 8 * (P.s - P.b);
  for (int l = 0; l < P.nlev; l++) {
    const int v0 = p.lev[l], v1 = p.lev[l + 1];
    const int sh = split ? 31 - __clz(max(step / (v1 - v0), 1)) : 0;  // (no level is empty)
    if (sh == 0) {
      for (int v = v0 + first; v < v1; v += step) {
        int32_t *q = st + v * kStripLd<CW> + c;
        int32_t acc = *q;
        const int e1 = p.eptr[v + 1];
#pragma unroll 4
        for (int i = p.eptr[v]; i < e1; i++) {
          const int2 x = p.ent[i];
          acc = __viaddmin_s32(x.y, st[x.x * kStripLd<CW> + c], acc);
        }
        *q = acc;
      }
    } else if (const int v = v0 + (first >> sh); v < v1) {
      int32_t acc = kInf;
      const int e1 = p.eptr[v + 1];
#pragma unroll 2
      for (int i = p.eptr[v] + (first & ((1 << sh) - 1)); i < e1; i += 1 << sh) {
        const int2 x = p.ent[i];
        acc = __viaddmin_s32(x.y, st[x.x * kStripLd<CW> + c], acc);
      }
      if (acc < kInf) atomicMin(st + v * kStripLd<CW> + c, acc);
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
template <int CW, bool SM>
__global__ void __launch_bounds__(kElimSweepThreads)
    elim_close_kernel(ElimDev e, const int32_t *__restrict__ list, const int64_t *__restrict__ out_off,
                      const int32_t *dB, int64_t ldB, int32_t *out, int64_t ld) {
  extern __shared__ __align__(16) int32_t st[];
  const ElimPart P = e.parts[list ? list[blockIdx.y] : blockIdx.y];
  const int x0 = blockIdx.x * CW;
  if (x0 >= P.s) return;
  const int nx = min(CW, P.s - x0);
  const int32_t *loc = e.loc + P.voff, *inv = e.inv + P.voff;
  const int c = threadIdx.x % CW, first = threadIdx.x / CW, step = blockDim.x / CW;
  const int lane = threadIdx.x & 31;
  const SweepPlan p = stage_plan<CW, SM>(e, P, st);
  for (int i = threadIdx.x; i < P.s * kStripLd<CW>; i += blockDim.x) st[i] = kInf;
  __syncthreads();
  for (int x = threadIdx.x >> 5; x < nx; x += blockDim.x >> 5) {
    int v = inv[x0 + x];
    if (lane == 0) st[v * kStripLd<CW> + x] = 0;
    __syncwarp();
    while (v >= P.b) {
      const int e0 = p.eptr[v], e1 = p.eptr[v + 1];
      if (e0 == e1) break;
      const int32_t y = st[v * kStripLd<CW> + x];
      const int up = p.ent[e0].x;
      if (y < kInf)
        for (int i = e0 + lane; i < e1; i += 32) {
          const int2 a = p.ent[i];
          int32_t *q = st + a.x * kStripLd<CW> + x;
          *q = __viaddmin_s32(a.y, y, *q);
        }
      __syncwarp();
      v = up;
    }
  }
  __syncthreads();
  if (P.b > 0) {
    for (int k = first; k < P.b; k += step) {
      const int32_t *row = dB + (int64_t)(P.boff + k) * ldB + P.boff;
      int32_t acc = st[k * kStripLd<CW> + c];
#pragma unroll 4
      for (int q = 0; q < P.b; q++) acc = __viaddmin_s32(__ldg(row + q), st[q * kStripLd<CW> + c], acc);
      st[k * kStripLd<CW> + c] = acc;
    }
    __syncthreads();
  }
  sweep_down<CW>(st, P, p);
  if (c < nx) {
    int32_t *o = out + out_off[blockIdx.y] + x0 + c;
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
  sweep_down<CW>(st, P, p);
  const int32_t *inv = e.inv + P.voff;
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < nr; r += blockDim.x >> 5) {
    int32_t *row = D + rows[2 * (r0 + r) + 1] * ldD;
    for (int i = lane; i < P.s; i += 32) row[vid[P.voff + i]] = st[inv[i] * kStripLd<CW> + r];
    if (blockIdx.y == 0)
      for (int64_t j = n + lane; j < ldD; j += 32) row[j] = kInf;
  }
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

cudaError_t launch_elim_up(const ElimDev &e, const int32_t *from, int32_t *M, int64_t ldM,
                           cudaStream_t stream, int64_t *launches) {
  if (e.nparts <= 0) return cudaSuccess;
  const size_t smem = (size_t)e.max_nent * sizeof(int2) + ((size_t)e.max_s + e.max_nlev + 2) * sizeof(int32_t);
  if (smem <= kElimSmem) {
    cudaError_t err = allow_smem(elim_up_kernel<true>, smem);
    if (err != cudaSuccess) return err;
    elim_up_kernel<true><<<e.nparts, kElimUpThreads, smem, stream>>>(e, from, M, ldM);
  } else {
    elim_up_kernel<false><<<e.nparts, kElimUpThreads, 0, stream>>>(e, from, M, ldM);
  }
  *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_elim_close(const ElimDev &e, const int32_t *list, const int64_t *out_off, int count, int max_s,
                              const int32_t *dB, int64_t ldB, int32_t *out, int64_t ld, cudaStream_t stream,
                              int64_t *launches) {
  if (count <= 0 || max_s <= 0) return cudaSuccess;
  return for_strip(e, max_s, [&](auto cw, auto sm) -> cudaError_t {
    constexpr int CW = decltype(cw)::value;
    constexpr bool SM = decltype(sm)::value;
    const size_t smem = sweep_bytes<CW>(e, max_s, SM);
    cudaError_t err = allow_smem(elim_close_kernel<CW, SM>, smem);
    if (err != cudaSuccess) return err;
    elim_close_kernel<CW, SM><<<dim3((max_s + CW - 1) / CW, count), kElimSweepThreads, smem, stream>>>(
        e, list, out_off, dB, ldB, out, ld);
    *launches += 1;
    return cudaGetLastError();
  });
}

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

}  // namespace fapb
