// Row sums of a 0/1 matrix over one base set by the MSM's bucket pipeline (zkb_msm.cu): the rows are
// taken `rho` at a time, a column's bits in such a group are a bucket number, every column is one mixed
// addition per group, and a row's sum is the sum of its group's buckets with its bit set.
#pragma once
#include <cstdint>

#include "zkb_runtime.h"

namespace zkb {

// Rows a group for launches of `ncols` columns and `nrows` rows, by field products: a mixed addition (10) for every
// column and group that is not all zeros, 2^(rho - 1) additions (16 lane products) for every row; few enough that the scan
// takes the buckets.
int msm_bits_group(int nrows, double ncols);
// Workspace bytes of a launch with exactly these sizes (a smaller one may need more).
zkg_status msm_bits_bytes(int curve, int nrows, int ncols, int rho, size_t* bytes);
// Enqueues the row sums of ncols columns (coeffs: row r at coeffs + r ld, non-zero bytes select) on st:
// row r's XYZZ point, canonical, goes to out + 4 r field elements, or with `add` is added to what is there.
// An error when ws_bytes is too small.
zkg_status msm_bits_launch(Context& cx, int curve, int nrows, int ncols, int rho, const uint8_t* coeffs, size_t ld,
                           const uint32_t* bases, char* ws, size_t ws_bytes, uint32_t* out, bool add,
                           cudaStream_t st);

}  // namespace zkb
