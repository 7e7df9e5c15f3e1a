// SELL-32 storage of a sparse matrix (host).
#ifndef SPG_SELL_BUILD_H
#define SPG_SELL_BUILD_H

#include <cstdint>
#include <vector>

namespace spg {

// CSR -> SELL-32 (slices of 32 rows, column-major, zero padding).
void build_sell32(int64_t n, const int32_t *row_ptr, const int32_t *col, const double *val,
                  std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol, std::vector<double> &sval);
void build_sell32(int64_t n, const int64_t *row_ptr, const int32_t *col, const double *val,
                  std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol, std::vector<double> &sval);
// Marks the banded slices of a square SELL-32 matrix: those whose entries fit
// into their width with entry j of lane l in column sref[j] + l, every such
// column of the 32 lanes inside the matrix. Their entries are reordered to that
// form (the columns of a row stay ascending; scol and sval stay a valid SELL-32
// matrix). stag: slice_ptr with bit 0 on a banded slice; sref: slice_ptr / 32
// words. Returns the number of banded slices.
int64_t band_sell32(int64_t n, const std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol,
                    std::vector<double> &sval, std::vector<int64_t> &stag, std::vector<int32_t> &sref);

}  // namespace spg

#endif
