// Floyd-Warshall closure of one matrix in pivot blocks of 64 (the form for
// matrices of up to some thousand vertices; launch_floyd_matrix chooses).
//
// One matrix leaves the chip idle between pivot blocks: with 128 x 128 tiles
// the diagonal tile (one CTA, 128 dependent pivots: 52 us), the panels (27 us)
// and the remainder (25 us at s = 1,500) follow one another, 105 us per block,
// while the relaxations of a block take 16 us at the DPX rate.  With blocks of
// 64 the diagonal tile takes an eighth of the work and every panel CTA closes
// it again for itself: two launches a block (panels 13 us, remainder 17 us at
// s = 1,500: 1,243 -> 731 us for the closure; 1,000: 833 -> 434).  With work
// space of its own a closure runs the panels beside the remainder of the block
// before them: one launch a block, 1,500: 731 -> 544, 1,000: 434 -> 343.  The
// two-launch form serves callers that have none (the plain form's parts and the
// allocation-free entry points).
#include <algorithm>
#include <type_traits>

#include "fap_common.cuh"
#include "fap_internal.h"
#include "floyd64_tiles.h"
#include "minplus_tile.cuh"

namespace fapb {
namespace {

constexpr int kB = 64;          // pivot block
constexpr int kThreads = 256;
constexpr int kLd = kB + 4;     // words between tile rows in shared memory: 16-byte aligned, the
                                // rows of a warp's two ty (one apart) in different banks

// Tile of `rows` x 64 from global memory into shared memory (row stride kLd).
template <typename T>
__device__ __forceinline__ void load_tile(T *dst, const T *src, int64_t ld, int rows) {
  using V = typename Vec4<T>::type;
  for (int t = threadIdx.x; t < rows * (kB / 4); t += kThreads) {
    const int r = t / (kB / 4), c = (t % (kB / 4)) * 4;
    *reinterpret_cast<V *>(dst + r * kLd + c) = *reinterpret_cast<const V *>(src + r * ld + c);
  }
}

// Closes the 64 x 64 tile at `src` into d (shared memory, stride kLd).  A
// thread holds 4 x 4 values; per pivot the owners publish row and column k,
// double-buffered, so one barrier per pivot.  A pivot row and column do not
// change in their own step (no negative entries).
template <typename T>
__device__ __forceinline__ void close_diag(const T *src, int64_t ld, T *d, T *line) {
  using V = typename Vec4<T>::type;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  T a[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const V v = *reinterpret_cast<const V *>(src + (4 * ty + i) * ld + 4 * tx);
    a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
  }
#pragma unroll 4
  for (int k = 0; k < kB; k++) {
    T *row = line + (k & 1) * 2 * kB, *col = row + kB;
    if (ty == k / 4) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i == (k & 3)) {
          V v;
          v.x = a[i][0]; v.y = a[i][1]; v.z = a[i][2]; v.w = a[i][3];
          *reinterpret_cast<V *>(row + 4 * tx) = v;
        }
    }
    if (tx == k / 4) {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j == (k & 3)) {
          V v;
          v.x = a[0][j]; v.y = a[1][j]; v.z = a[2][j]; v.w = a[3][j];
          *reinterpret_cast<V *>(col + 4 * ty) = v;
        }
    }
    __syncthreads();
    const V r4 = *reinterpret_cast<const V *>(row + 4 * tx), c4 = *reinterpret_cast<const V *>(col + 4 * ty);
    const T r[4] = {r4.x, r4.y, r4.z, r4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) a[i][j] = Dist<T>::relax(c[i], r[j], a[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    V v;
    v.x = a[i][0]; v.y = a[i][1]; v.z = a[i][2]; v.w = a[i][3];
    *reinterpret_cast<V *>(d + (4 * ty + i) * kLd + 4 * tx) = v;
  }
}

// acc(r, c) <- min(acc, min_k A[r][k] + B[k][c]) over 64 k, rows r = ty + 16 i,
// columns 4 tx + j, both tiles in shared memory.
template <typename T, int NR>
__device__ __forceinline__ void product64(const T *A, const T *B, T (&acc)[NR][4]) {
  using V = typename Vec4<T>::type;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll 4
  for (int k = 0; k < kB; k += 4) {
    T a[NR][4];
#pragma unroll
    for (int i = 0; i < NR; i++) {
      const V v = *reinterpret_cast<const V *>(A + (ty + 16 * i) * kLd + k);
      a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const V v = *reinterpret_cast<const V *>(B + (k + q) * kLd + 4 * tx);
      const T b[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < NR; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = Dist<T>::relax(a[i][q], b[j], acc[i][j]);
    }
  }
}

template <typename T, int NR>
__device__ __forceinline__ void load_acc(T (&acc)[NR][4], const T *tile) {
  using V = typename Vec4<T>::type;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < NR; i++) {
    const V v = *reinterpret_cast<const V *>(tile + (ty + 16 * i) * kLd + 4 * tx);
    acc[i][0] = v.x; acc[i][1] = v.y; acc[i][2] = v.z; acc[i][3] = v.w;
  }
}

template <typename T>
__device__ __forceinline__ void store_row(T *dst, const T (&a)[4]) {
  typename Vec4<T>::type v;
  v.x = a[0]; v.y = a[1]; v.z = a[2]; v.w = a[3];
  *reinterpret_cast<typename Vec4<T>::type *>(dst) = v;
}

// A 64 x 64 tile held as acc (rows ty + 16 i) also stored transposed at dst,
// through shared memory (buf: kB x kLd words, free for this use).
template <typename T, int NR>
__device__ __forceinline__ void store_transposed(const T (&acc)[NR][4], int i0, T *buf, T *dst, int64_t ld) {
  using V = typename Vec4<T>::type;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) buf[(4 * tx + j) * kLd + ty + 16 * i] = acc[i0 + i][j];
  __syncthreads();
  for (int t = threadIdx.x; t < kB * (kB / 4); t += kThreads) {
    const int r = t / (kB / 4), c = (t % (kB / 4)) * 4;
    *reinterpret_cast<V *>(dst + r * ld + c) = *reinterpret_cast<const V *>(buf + r * kLd + c);
  }
}

// Panels of pivot block kb: CTA x < nb - 1 the row panel's tile, then (not
// SYM) the column panel's; SYM also stores the row panel's transposes.
template <typename T, bool SYM>
__global__ void __launch_bounds__(kThreads) floyd64_panel_kernel(T *mat, int64_t ld, int kb, int nb) {
  __shared__ __align__(16) T diag[kB * kLd], tile[kB * kLd], line[4 * kB];
  const bool row = (int)blockIdx.x < nb - 1;
  int t = row ? blockIdx.x : blockIdx.x - (nb - 1);
  t += t >= kb;
  const T *D = mat + (int64_t)kb * kB * (ld + 1);
  T *P = row ? mat + (int64_t)kb * kB * ld + (int64_t)t * kB : mat + (int64_t)t * kB * ld + (int64_t)kb * kB;
  load_tile(tile, P, ld, kB);
  close_diag(D, ld, diag, line);
  __syncthreads();
  T acc[4][4];
  load_acc(acc, tile);
  if (row) product64<T, 4>(diag, tile, acc);
  else product64<T, 4>(tile, diag, acc);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
#pragma unroll
  for (int i = 0; i < 4; i++) store_row(P + (ty + 16 * i) * ld + 4 * tx, acc[i]);
  if (SYM) store_transposed<T, 4>(acc, 0, tile, mat + (int64_t)t * kB * ld + (int64_t)kb * kB, ld);
}

// Remainder tiles (i0, jx) and (i0 + 1, jx) of pivot block kb, as far as they
// are this CTA's (floyd64_pair_rows), of nr rows and columns counted without the
// `skip` ones from kb on.  SYM: each is also stored transposed.
template <typename T, bool SYM>
__device__ __forceinline__ void rest_tiles(T *mat, int64_t ld, int kb, int jx, int i0, int nr, int skip, T *A, T *B) {
  const int ni = floyd64_pair_rows(SYM, jx, i0, nr);
  if (ni == 0) return;
  const int j = jx + (jx >= kb ? skip : 0);
  const int ia = i0 + (i0 >= kb ? skip : 0), ib = ni > 1 ? i0 + 1 + (i0 + 1 >= kb ? skip : 0) : ia;
  const T *R = mat + (int64_t)kb * kB * ld + (int64_t)j * kB;
  load_tile(A, mat + (int64_t)ia * kB * ld + (int64_t)kb * kB, ld, kB);
  load_tile(A + kB * kLd, mat + (int64_t)ib * kB * ld + (int64_t)kb * kB, ld, kB);
  load_tile(B, R, ld, kB);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  T *Ca = mat + (int64_t)ia * kB * ld + (int64_t)j * kB, *Cb = mat + (int64_t)ib * kB * ld + (int64_t)j * kB;
  using V = typename Vec4<T>::type;
  T acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const V v = *reinterpret_cast<const V *>((i < 4 ? Ca + (ty + 16 * i) * ld : Cb + (ty + 16 * (i - 4)) * ld) + 4 * tx);
    acc[i][0] = v.x; acc[i][1] = v.y; acc[i][2] = v.z; acc[i][3] = v.w;
  }
  __syncthreads();
  product64<T, 8>(A, B, acc);
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (i < 4 || ni > 1)
      store_row((i < 4 ? Ca + (ty + 16 * i) * ld : Cb + (ty + 16 * (i - 4)) * ld) + 4 * tx, acc[i]);
  if (SYM) {
    if (ia != j) store_transposed<T, 8>(acc, 0, A, mat + (int64_t)j * kB * ld + (int64_t)ia * kB, ld);
    if (ni > 1 && ib != j) store_transposed<T, 8>(acc, 4, A, mat + (int64_t)j * kB * ld + (int64_t)ib * kB, ld);
  }
}

// Remainder of pivot block kb: CTA (column tile, pair of row tiles) of the
// tiles outside the pivot's row and column; the last CTA of x = 0 closes the
// diagonal tile in place (the panels closed it for themselves).  SYM: only row
// tiles up to the column tile, each also stored transposed.  CTAS: per SM; a
// grid of more than two waves takes three at 80 registers (s = 4,000 6.19 ->
// 5.69 ms; symmetric 5,538 12.1 -> 10.9), a smaller one two without spills
// (1,500 732 us, 784 with three).
template <typename T, bool SYM, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS) floyd64_rest_kernel(T *mat, int64_t ld, int kb, int nb) {
  extern __shared__ __align__(16) unsigned char f64_smem[];
  T *A = reinterpret_cast<T *>(f64_smem), *B = A + 2 * kB * kLd;
  if (blockIdx.y == gridDim.y - 1) {
    if (blockIdx.x != 0) return;
    T *D = mat + (int64_t)kb * kB * (ld + 1);
    close_diag(D, ld, A, B);
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    T acc[4][4];
    load_acc(acc, A);
#pragma unroll
    for (int i = 0; i < 4; i++) store_row(D + (ty + 16 * i) * ld + 4 * tx, acc[i]);
    return;
  }
  rest_tiles<T, SYM>(mat, ld, kb, blockIdx.x, 2 * blockIdx.y, nb - 1, 1, A, B);
}

// Panel tile of pivot block nx (tile t of its row, or of its column) while the
// remainder of the block before it, kb = nx - 1, is still running: the tile and
// the diagonal tile take kb's product here first.  No CTA of the launch writes
// what another reads: the corner tiles (nx, kb) and (kb, nx), operands of all
// panels and themselves panels of nx, are read as copies that the launch before
// left in `work`; the closed diagonal tile goes to `work` and into the matrix
// with the next launch.  work: per parity of the pivot block the copies of
// (k + 1, k) and (k, k + 1) and the closed tile (k, k), rows of 64 words.
template <typename T, bool SYM>
__device__ __forceinline__ void panel_ahead(T *mat, int64_t ld, int nx, int nb, int x, T *work, T *A, T *B) {
  using V = typename Vec4<T>::type;
  T *A1 = A + kB * kLd, *line = B + kB * kLd;
  const int kb = nx - 1;
  const bool row = x < nb - 1;
  int t = row ? x : x - (nb - 1);
  t += t >= nx;
  const T *D = mat + (int64_t)nx * kB * (ld + 1);
  T *P = row ? mat + (int64_t)nx * kB * ld + (int64_t)t * kB : mat + (int64_t)t * kB * ld + (int64_t)nx * kB;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  T acc[4][4], dg[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const V v = *reinterpret_cast<const V *>(P + (ty + 16 * i) * ld + 4 * tx);
    acc[i][0] = v.x; acc[i][1] = v.y; acc[i][2] = v.z; acc[i][3] = v.w;
    const V u = *reinterpret_cast<const V *>(D + (ty + 16 * i) * ld + 4 * tx);
    dg[i][0] = u.x; dg[i][1] = u.y; dg[i][2] = u.z; dg[i][3] = u.w;
  }
  if (kb >= 0) {
    const T *S = work + (kb & 1) * 3 * kB * kB;
    load_tile(A, S, kB, kB);
    load_tile(A1, S + kB * kB, kB, kB);
    if (t != kb)  // (a tile of kb's own panels is final for kb)
      load_tile(B, row ? mat + (int64_t)kb * kB * ld + (int64_t)t * kB : mat + (int64_t)t * kB * ld + (int64_t)kb * kB,
                ld, kB);
    __syncthreads();
    product64<T, 4>(A, A1, dg);
    if (t != kb) {
      if (row) product64<T, 4>(A, B, acc);
      else product64<T, 4>(B, A1, acc);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    store_row(A + (ty + 16 * i) * kLd + 4 * tx, dg[i]);
    store_row(B + (ty + 16 * i) * kLd + 4 * tx, acc[i]);
  }
  __syncthreads();
  close_diag(A, kLd, A1, line);
  __syncthreads();
  if (row) product64<T, 4>(A1, B, acc);
  else product64<T, 4>(B, A1, acc);
  T *W = work + (nx & 1) * 3 * kB * kB;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    store_row(P + (ty + 16 * i) * ld + 4 * tx, acc[i]);
    if (t == nx + 1) store_row(W + (row ? kB * kB : 0) + (ty + 16 * i) * kB + 4 * tx, acc[i]);
  }
  if (x == 0)
    for (int q = threadIdx.x; q < kB * (kB / 4); q += kThreads) {
      const int r = q / (kB / 4), c = (q % (kB / 4)) * 4;
      *reinterpret_cast<V *>(W + 2 * kB * kB + r * kB + c) = *reinterpret_cast<const V *>(A1 + r * kLd + c);
    }
  if (SYM) {
    store_transposed<T, 4>(acc, 0, A, mat + (int64_t)t * kB * ld + (int64_t)nx * kB, ld);
    if (t == nx + 1) store_transposed<T, 4>(acc, 0, A, W, kB);
  }
}

// One launch per pivot block: the panels of block kb + 1 (first in the grid)
// beside the remainder of block kb, which is the tiles outside rows and columns
// kb and kb + 1.  A panel is a chain of some 13 us whatever the matrix, so the
// launches for panels and remainders one after the other left the chip idle for
// nearly as long again as the remainder takes at s = 1,500; kb = -1 starts the
// chain.  int32, us, two launches / one: s = 500 211 / 185, 1,000 434 / 343,
// 1,500 731 / 544, 4,000 5,690 / 5,420.  CTAS: as for floyd64_rest_kernel.
template <typename T, bool SYM, int CTAS>
__global__ void __launch_bounds__(kThreads, CTAS) floyd64_step_kernel(T *mat, int64_t ld, int kb, int nb, T *work) {
  extern __shared__ __align__(16) unsigned char f64_smem[];
  T *A = reinterpret_cast<T *>(f64_smem), *B = A + 2 * kB * kLd;
  const bool last = kb + 1 == nb;
  const int np = last ? 0 : (SYM ? 1 : 2) * (nb - 1);
  if ((int)blockIdx.x < np) {
    panel_ahead<T, SYM>(mat, ld, kb + 1, nb, blockIdx.x, work, A, B);
    return;
  }
  const int id = blockIdx.x - np - 1, skip = last ? 1 : 2, nr = nb - skip;
  if (id < 0) {  // the closed diagonal tile
    using V = typename Vec4<T>::type;
    const T *S = work + ((kb & 1) * 3 + 2) * kB * kB;
    T *D = mat + (int64_t)kb * kB * (ld + 1);
    for (int q = threadIdx.x; q < kB * (kB / 4); q += kThreads) {
      const int r = q / (kB / 4), c = (q % (kB / 4)) * 4;
      *reinterpret_cast<V *>(D + r * ld + c) = *reinterpret_cast<const V *>(S + r * kB + c);
    }
    return;
  }
  rest_tiles<T, SYM>(mat, ld, kb, id % nr, 2 * (id / nr), nr, skip, A, B);
}

template <typename T, bool SYM>
cudaError_t run(T *mat, int64_t ld, int nb, T *work, cudaStream_t stream, int64_t *launches) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = ((size_t)3 * kB * kLd + 4 * kB) * sizeof(T);
  const bool many = (int64_t)(nb - 1) * (nb / 2) / (SYM ? 2 : 1) > 4 * (int64_t)sms;
  if (work && nb > 1) {
    auto step = many ? floyd64_step_kernel<T, SYM, 3> : floyd64_step_kernel<T, SYM, 2>;
    cudaError_t e = cudaFuncSetAttribute(step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int np = (SYM ? 1 : 2) * (nb - 1);
    for (int kb = -1; kb < nb; kb++) {
      const int nr = kb + 1 < nb ? nb - 2 : nb - 1;
      const int grid = kb < 0 ? np : (kb + 1 < nb ? np : 0) + 1 + nr * ((nr + 1) / 2);
      step<<<grid, kThreads, smem, stream>>>(mat, ld, kb, nb, work);
      *launches += 1;
    }
    return cudaGetLastError();
  }
  auto rest = many ? floyd64_rest_kernel<T, SYM, 3> : floyd64_rest_kernel<T, SYM, 2>;
  cudaError_t e = cudaFuncSetAttribute(rest, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  for (int kb = 0; kb < nb; kb++) {
    if (nb > 1) {
      floyd64_panel_kernel<T, SYM><<<(SYM ? 1 : 2) * (nb - 1), kThreads, 0, stream>>>(mat, ld, kb, nb);
      *launches += 1;
    }
    rest<<<dim3(std::max(1, nb - 1), nb / 2 + 1), kThreads, smem, stream>>>(mat, ld, kb, nb);
    *launches += 1;
  }
  return cudaGetLastError();
}

template <typename T>
__global__ void pad_copy_kernel(T *dst, int64_t ldd, const T *__restrict__ src, int64_t lds, int s) {
  using V = typename Vec4<T>::type;
  for (int64_t i = blockIdx.y; i < ldd; i += gridDim.y)
    for (int64_t j = 4 * (blockIdx.x * (int64_t)blockDim.x + threadIdx.x); j < ldd;
         j += 4 * (int64_t)gridDim.x * blockDim.x) {
      T a[4];
#pragma unroll
      for (int q = 0; q < 4; q++) a[q] = i < s && j + q < s ? __ldg(src + i * lds + j + q) : Dist<T>::inf();
      V v;
      v.x = a[0]; v.y = a[1]; v.z = a[2]; v.w = a[3];
      *reinterpret_cast<V *>(dst + i * ldd + j) = v;
    }
}

}  // namespace

template <typename T>
cudaError_t launch_pad_copy(T *dst, int64_t ldd, const T *src, int64_t lds, int s, cudaStream_t stream,
                            int64_t *launches) {
  const dim3 grid((unsigned)ceil_div(ldd, 4 * kThreads), (unsigned)std::min<int64_t>(ldd, kMaxGridY));
  pad_copy_kernel<T><<<grid, kThreads, 0, stream>>>(dst, ldd, src, lds, s);
  *launches += 1;
  return cudaGetLastError();
}
template cudaError_t launch_pad_copy<int32_t>(int32_t *, int64_t, const int32_t *, int64_t, int, cudaStream_t, int64_t *);
template cudaError_t launch_pad_copy<float>(float *, int64_t, const float *, int64_t, int, cudaStream_t, int64_t *);

// mat: rows and columns up to the next multiple of 64 hold the sentinel.
template <typename T>
cudaError_t launch_floyd64(T *mat, int64_t ld, int s, bool sym, T *work, cudaStream_t stream, int64_t *launches) {
  static_assert(kFloyd64Work == 6 * kB * kB, "two parities of three tiles");
  const int nb = (int)ceil_div(s, kB);
  if (ld % 4 != 0 || (int64_t)nb * kB > ld) return cudaErrorInvalidValue;
  return sym ? run<T, true>(mat, ld, nb, work, stream, launches) : run<T, false>(mat, ld, nb, work, stream, launches);
}
template cudaError_t launch_floyd64<int32_t>(int32_t *, int64_t, int, bool, int32_t *, cudaStream_t, int64_t *);
template cudaError_t launch_floyd64<float>(float *, int64_t, int, bool, float *, cudaStream_t, int64_t *);

}  // namespace fapb
