// rb_index.h -- element offsets of realqm_rb.js fields: from NN = 1290 on a field has more than 2^31 elements
// (two electrons there are 65 GB), from NN = 1627 its interior more than 2^32.
#pragma once

#ifdef __CUDACC__
#define RQ_RB_HD __host__ __device__ __forceinline__
#else
#define RQ_RB_HD inline
#endif

namespace rq {

// The kernels come in both widths of I: 64-bit offsets throughout cost H2 at 100^3 4-8 % (3.61 ms a case, 3.73
// to 3.90).  A 32-bit I only where this holds: there also a walk's next strides (8 x 256 x 128 cells) stay below 2^32.
RQ_RB_HD bool rb_offsets_fit_31_bits(int NN) { return NN <= 1289; }

template <typename I>
RQ_RB_HD I rb_offset(int i, int j, int k, int S) {
  return (I)i * (S * S) + (I)j * S + k;
}

// offset of interior cell number `cell` (k fastest, NM = NN - 1 cells a side)
template <typename I>
RQ_RB_HD I rb_interior_offset(I cell, int NM, int S) {
  const I n = (I)NM, s = (I)S, y = cell / n, k = cell - y * n, i = y / n, j = y - i * n;
  return ((i + 1) * s + j + 1) * s + k + 1;
}

}  // namespace rq
