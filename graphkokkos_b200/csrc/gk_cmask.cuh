// Internal interface of the complement-masked product's sorting path (cmask_sort.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gk_common.cuh"

namespace gk {

// C<!M> = A·B by expanding, sorting and reducing the products.  work: products of
// every row (device); each below 2^31.  Without c_col cnt[0, m) receives the rows'
// entries.  With it (and crp, C's row pointers in device memory) the columns and
// values (c_val may be null) are written, and *mismatch is set where crp is not
// this product's; nothing is written beyond the crp[m] entries.
int cmask_by_sort(const DevCsr &a, const DevCsr &b, const DevCsr &mk, bool values, const int64_t *work, int64_t *cnt,
                  const int64_t *crp, int32_t *c_col, int32_t *c_val, unsigned int *mismatch, cudaStream_t s,
                  Scratch &scr);

}  // namespace gk
