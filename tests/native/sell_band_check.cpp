// Banded slices of SELL-32 (sell_build.h) against the CSR matrix: for several
// orderings and sizes prints "slices banded wrong", wrong counting the rows
// whose entries, read by either form, are not the row's.
#include <algorithm>
#include <cstdio>
#include <map>
#include <random>

#include "../../start_gb300/csrc/sell_build.h"

using namespace spg;

struct Csr {
    int64_t n;
    std::vector<int64_t> rp;
    std::vector<int32_t> ci;
    std::vector<double> v;
};

// Lattice of nx x ny x nz nodes with 7 or 15 couplings per node, every `cut`-th
// row the identity, nodes renumbered by perm.
static Csr lattice(int nx, int ny, int nz, bool wide, int cut, const std::vector<int32_t> &perm, std::mt19937 &g) {
    Csr A;
    A.n = int64_t(nx) * ny * nz;
    std::vector<std::map<int32_t, double>> rows(A.n);
    std::uniform_real_distribution<double> u(0.5, 1.5);
    for (int z = 0; z < nz; ++z)
        for (int y = 0; y < ny; ++y)
            for (int x = 0; x < nx; ++x) {
                const int32_t i = perm[(int64_t(z) * ny + y) * nx + x];
                rows[i][i] = 7.0;
                if (cut && i % cut == 0) continue;
                for (int d = 1; d < 8; ++d)
                    for (int s = -1; s <= 1; s += 2) {
                        const int dx = d & 1, dy = (d >> 1) & 1, dz = d >> 2;
                        if (!wide && dx + dy + dz > 1) continue;
                        const int a = x + s * dx, b = y + s * dy, c = z + s * dz;
                        if (a < 0 || b < 0 || c < 0 || a >= nx || b >= ny || c >= nz) continue;
                        rows[i][perm[(int64_t(c) * ny + b) * nx + a]] = d == 5 ? 0.0 : -u(g);  // exact zeros too
                    }
            }
    A.rp.push_back(0);
    for (auto &r : rows) {
        for (auto &e : r) {
            A.ci.push_back(e.first);
            A.v.push_back(e.second);
        }
        A.rp.push_back(int64_t(A.ci.size()));
    }
    return A;
}

static void check(const Csr &A) {
    std::vector<int64_t> sp, tag;
    std::vector<int32_t> sc, ref;
    std::vector<double> sv;
    build_sell32(A.n, A.rp.data(), A.ci.data(), A.v.data(), sp, sc, sv);
    const auto sp0 = sp;
    const int64_t banded = band_sell32(A.n, sp, sc, sv, tag, ref);
    int64_t wrong = sp == sp0 ? 0 : 1, marked = 0;
    for (size_t s = 0; s + 1 < sp.size(); ++s) marked += tag[s] & 1;
    wrong += marked == banded ? 0 : 1;
    for (int64_t i = 0; i < 32 * (int64_t(sp.size()) - 1); ++i) {
        const int64_t s = i / 32, l = i % 32, w = (sp[s + 1] - sp[s]) / 32;
        std::map<int32_t, double> want, plain, band;
        if (i < A.n)
            for (int64_t k = A.rp[i]; k < A.rp[i + 1]; ++k)
                if (A.v[k] != 0.0) want[A.ci[k]] = A.v[k];
        bool in = true;
        for (int64_t j = 0; j < w; ++j) {
            const int64_t o = sp[s] + 32 * j + l;
            in = in && sc[o] >= 0 && sc[o] < A.n;
            if (sv[o] != 0.0) plain[sc[o]] += sv[o];
            const int64_t c = (tag[s] & 1) ? ref[size_t(sp[s] / 32 + j)] + l : sc[o];
            in = in && c >= 0 && c < A.n;
            if (sv[o] != 0.0) band[int32_t(c)] += sv[o];
        }
        wrong += in && plain == want && band == want ? 0 : 1;
    }
    std::printf("%lld %lld %lld\n", (long long)(sp.size() - 1), (long long)banded, (long long)wrong);
}

int main() {
    std::mt19937 g(5);
    const int dims[][3] = {{1, 1, 1}, {2, 3, 4}, {31, 4, 3}, {32, 5, 4}, {33, 5, 4}, {101, 7, 5}, {7, 9, 11}, {64, 8, 2}};
    for (auto &d : dims)
        for (int wide = 0; wide < 2; ++wide)
            for (int order = 0; order < 3; ++order) {
                const int64_t n = int64_t(d[0]) * d[1] * d[2];
                std::vector<int32_t> perm(n);
                for (int64_t i = 0; i < n; ++i) perm[i] = int32_t(i);
                if (order == 1) std::shuffle(perm.begin(), perm.end(), g);
                if (order == 2) std::reverse(perm.begin(), perm.end());
                check(lattice(d[0], d[1], d[2], wide, order == 2 ? 5 : 0, perm, g));
            }
    return 0;
}
