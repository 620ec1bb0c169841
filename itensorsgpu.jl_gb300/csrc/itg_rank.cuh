// The order of singular and eigenvalues, shared by every ranking kernel (plain C++ as well).
#pragma once

#ifdef __CUDACC__
#define ITG_RANK_FN __host__ __device__ __forceinline__
#else
#define ITG_RANK_FN inline
#endif

// Whether value i (u) ranks before value j (v): descending, ties by index, NaN
// before every number (so that a caller sees it, as the first value, however
// much is truncated).  A total order: the ranks of any n values are 0 .. n - 1, each
// once.  The gathers read columns through the ranks, so every slot must be
// written whatever the values are.
ITG_RANK_FN bool itg_rank_before(double u, int i, double v, int j) {
  const bool un = u != u, vn = v != v;
  if (un || vn) return un && (!vn || i < j);
  return u > v || (u == v && i < j);
}
