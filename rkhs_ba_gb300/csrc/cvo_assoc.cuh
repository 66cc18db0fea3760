// cvo_assoc.cuh -- the instances of the association kernels for one label stride.
//
// Feature rows are stored as ceil(F/4) float4 chunks, label rows as 5 or 9 chunks (C <= 20 or
// C <= 36, padded at upload).  One translation unit per label stride: they compile in parallel.
#pragma once
#include "cvo_kernels.cuh"

namespace cvo_gb {

template <int FC, int LC, bool G>
inline int assoc_instances(AssocKernels *a) {
  a->cand = k_cand<FC>;
  a->rows[ROWS_ALL] = k_rows<FC, LC, G, ROWS_SUM, ROWS_ALL>;
  a->rows[ROWS_LIGHT] = k_rows<FC, LC, G, ROWS_SUM, ROWS_LIGHT>;
  a->ordered_rows[ROWS_ALL] = k_rows<FC, LC, G, ROWS_ORDERED, ROWS_ALL>;
  a->ordered_rows[ROWS_LIGHT] = k_rows<FC, LC, G, ROWS_ORDERED, ROWS_LIGHT>;
  return 0;
}

template <int LC>
inline int assoc_kernels(int fch, bool gt, AssocKernels *a) {
  if (fch == 0) return gt ? assoc_instances<0, LC, true>(a) : assoc_instances<0, LC, false>(a);
  if (fch == 1) return gt ? assoc_instances<1, LC, true>(a) : assoc_instances<1, LC, false>(a);
  return gt ? assoc_instances<2, LC, true>(a) : assoc_instances<2, LC, false>(a);
}

}  // namespace cvo_gb
