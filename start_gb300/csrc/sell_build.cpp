#include "sell_build.h"

#include <algorithm>

namespace spg {

// Entries that are exactly zero off the diagonal are left out (the P1
// stiffness of a Kuhn-split lattice is the 7-point stencil: 8 of its 15
// structural couplings per row are exact zeros); a product with an exact
// zero adds nothing to a sum, so A x is unchanged.
template <class RP>
static void build_sell32_t(int64_t n, const RP *row_ptr, const int32_t *col, const double *val,
                           std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol, std::vector<double> &sval) {
    auto kept = [&](int64_t r, int64_t k) { return val[k] != 0.0 || col[k] == r; };
    const int64_t ns = (n + 31) / 32;
    slice_ptr.assign(ns + 1, 0);
#pragma omp parallel for schedule(static)
    for (int64_t sl = 0; sl < ns; ++sl) {
        int64_t w = 0;
        for (int64_t r = sl * 32; r < std::min(n, sl * 32 + 32); ++r) {
            int64_t len = 0;
            for (int64_t k = int64_t(row_ptr[r]); k < int64_t(row_ptr[r + 1]); ++k) len += kept(r, k) ? 1 : 0;
            w = std::max(w, len);
        }
        slice_ptr[sl + 1] = 32 * w;
    }
    for (int64_t sl = 0; sl < ns; ++sl) slice_ptr[sl + 1] += slice_ptr[sl];
    scol.resize(slice_ptr[ns]);
    sval.resize(slice_ptr[ns]);
#pragma omp parallel for schedule(static)
    for (int64_t sl = 0; sl < ns; ++sl) {
        const int64_t w = (slice_ptr[sl + 1] - slice_ptr[sl]) / 32;
        for (int64_t l = 0; l < 32; ++l) {
            const int64_t r = sl * 32 + l;
            int64_t j = 0;
            int32_t first = 0;
            if (r < n)
                for (int64_t k = int64_t(row_ptr[r]); k < int64_t(row_ptr[r + 1]); ++k) {
                    if (!kept(r, k)) continue;
                    const int64_t o = slice_ptr[sl] + 32 * j + l;
                    scol[o] = col[k];
                    sval[o] = val[k];
                    if (j == 0) first = col[k];
                    ++j;
                }
            // padding: value 0 at a column the row already reads (or column
            // 0), always inside x also for a rectangular matrix
            for (; j < w; ++j) {
                const int64_t o = slice_ptr[sl] + 32 * j + l;
                scol[o] = first;
                sval[o] = 0.0;
            }
        }
    }
}

void build_sell32(int64_t n, const int32_t *row_ptr, const int32_t *col, const double *val,
                  std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol, std::vector<double> &sval) {
    build_sell32_t(n, row_ptr, col, val, slice_ptr, scol, sval);
}
void build_sell32(int64_t n, const int64_t *row_ptr, const int32_t *col, const double *val,
                  std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol, std::vector<double> &sval) {
    build_sell32_t(n, row_ptr, col, val, slice_ptr, scol, sval);
}

int64_t band_sell32(int64_t n, const std::vector<int64_t> &slice_ptr, std::vector<int32_t> &scol,
                    std::vector<double> &sval, std::vector<int64_t> &stag, std::vector<int32_t> &sref) {
    constexpr int kWidest = 64;  // wider slices are left as they are
    const int64_t ns = int64_t(slice_ptr.size()) - 1;
    stag = slice_ptr;
    sref.assign(size_t(slice_ptr[ns] / 32), 0);
    int64_t banded = 0;
#pragma omp parallel for schedule(static) reduction(+ : banded)
    for (int64_t sl = 0; sl < ns; ++sl) {
        const int64_t base = slice_ptr[sl];
        const int w = int((slice_ptr[sl + 1] - base) / 32);
        if (w == 0 || w > kWidest) continue;
        const int rows = int(std::min<int64_t>(32, n - sl * 32));
        // padding has value 0 and is not the row's (first) diagonal entry, the
        // only zero that build_sell32 keeps; before: the row's last column so far
        auto pad = [&](int64_t o, int l, int64_t before) {
            return sval[o] == 0.0 && (scol[o] != sl * 32 + l || scol[o] <= before);
        };
        int64_t refs[kWidest + 1];
        int nr = 0;
        bool ok = true;
        for (int l = 0; l < rows && ok; ++l) {
            int64_t before = -1;
            int at = 0;  // refs[at - 1] < the row's next reference
            for (int j = 0; j < w && ok; ++j) {
                const int64_t o = base + 32 * j + l;
                if (pad(o, l, before)) continue;
                ok = scol[o] > before;
                before = scol[o];
                const int64_t ref = int64_t(scol[o]) - l;
                while (at < nr && refs[at] < ref) ++at;
                if (at == nr || refs[at] != ref) {
                    if (nr == w) {
                        ok = false;
                        break;
                    }
                    for (int k = nr; k > at; --k) refs[k] = refs[k - 1];
                    refs[at] = ref;
                    ++nr;
                }
            }
        }
        if (!ok || nr == 0 || refs[0] < 0 || refs[nr - 1] + 31 >= n) continue;
        for (int l = 0; l < 32; ++l) {
            int32_t c[kWidest];
            double v[kWidest];
            int m = 0;
            const int32_t first = scol[base + l];
            if (l < rows)
                for (int j = 0; j < w; ++j) {
                    const int64_t o = base + 32 * j + l;
                    if (pad(o, l, m ? c[m - 1] : -1)) continue;
                    c[m] = scol[o];
                    v[m++] = sval[o];
                }
            int k = 0;
            for (int j = 0; j < w; ++j) {
                const int64_t o = base + 32 * j + l;
                const bool here = k < m && j < nr && c[k] - l == refs[j];
                scol[o] = here ? c[k] : first;
                sval[o] = here ? v[k] : 0.0;
                k += here ? 1 : 0;
            }
        }
        for (int j = 0; j < w; ++j) sref[size_t(base / 32 + j)] = int32_t(refs[std::min(j, nr - 1)]);
        stag[sl] |= 1;
        ++banded;
    }
    return banded;
}

}  // namespace spg
