// Which tiles a CTA of the blocks-of-64 Floyd remainder takes (fap_floyd64.cu).
// Plain C++, so that the cover can be checked on the host.
#pragma once

#if defined(__CUDACC__)
#define FAPB_HD __host__ __device__
#else
#define FAPB_HD
#endif

namespace fapb {

// Rows of the pair (i0, i0 + 1) that the CTA of column jx (both counted without
// the pivot's rows and columns, nr of them) takes.  sym: only rows up to the
// column's, each also stored transposed, so that no tile has two writers: the
// tile below the diagonal at (jx + 1, jx) comes from column jx + 1.
FAPB_HD inline int floyd64_pair_rows(bool sym, int jx, int i0, int nr) {
  int ni = nr - i0 < 2 ? nr - i0 : 2;
  if (sym && i0 + ni - 1 > jx) ni = jx - i0 + 1;
  return ni > 0 ? ni : 0;
}

}  // namespace fapb
