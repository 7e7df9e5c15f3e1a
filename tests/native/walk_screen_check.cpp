// The FP32-screened walk decision (screen.h) against the FP64 evaluation of
// the walk on random tets: prints "decided undecided wrong" per kind of case.
// The FP64 side evaluates the expressions of the oracle's walk in their order
// (built with -ffp-contract=off).
#include <cmath>
#include <cstdio>
#include <random>

#include "../../start_gb300/csrc/screen.h"

using namespace spg;

struct Tet {
    double M[9], x0[3];
    float Mf[9];
};

static Tet make(const double v[4][3]) {
    double J[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) J[3 * c + r] = v[r + 1][c] - v[0][c];  // columns: edges
    const double det = J[0] * (J[4] * J[8] - J[5] * J[7]) - J[1] * (J[3] * J[8] - J[5] * J[6]) +
                       J[2] * (J[3] * J[7] - J[4] * J[6]);
    Tet t;
    const double adj[9] = {J[4] * J[8] - J[5] * J[7], J[2] * J[7] - J[1] * J[8], J[1] * J[5] - J[2] * J[4],
                           J[5] * J[6] - J[3] * J[8], J[0] * J[8] - J[2] * J[6], J[2] * J[3] - J[0] * J[5],
                           J[3] * J[7] - J[4] * J[6], J[1] * J[6] - J[0] * J[7], J[0] * J[4] - J[1] * J[3]};
    for (int k = 0; k < 9; ++k) {
        t.M[k] = adj[k] / det;
        t.Mf[k] = hi_float(t.M[k]);
    }
    for (int k = 0; k < 3; ++k) t.x0[k] = v[0][k];
    return t;
}

static void bary(const Tet &t, const double p[3], double l[4]) {
    const double d0 = p[0] - t.x0[0], d1 = p[1] - t.x0[1], d2 = p[2] - t.x0[2];
    l[1] = t.M[0] * d0 + t.M[1] * d1 + t.M[2] * d2;
    l[2] = t.M[3] * d0 + t.M[4] * d1 + t.M[5] * d2;
    l[3] = t.M[6] * d0 + t.M[7] * d1 + t.M[8] * d2;
    l[0] = 1.0 - l[1] - l[2] - l[3];
}

static int exact(const Tet &t, const double p0[3], const double p1[3], int enter) {
    double l1[4], l0[4];
    bary(t, p1, l1);
    bary(t, p0, l0);
    int best = -1, n = 0;
    double sb = 0.0;
    for (int f = 0; f < 4; ++f) n += f != enter && l1[f] < 0.0;
    if (n == 0) return kScreenInside;
    for (int f = 0; f < 4; ++f) {
        if (f == enter || !(l1[f] < 0.0)) continue;
        const double s = l0[f] / (l0[f] - l1[f]);
        if (best < 0 || s < sb) {
            best = f;
            sb = s;
        }
    }
    return best;
}

int main() {
    std::mt19937_64 g(12345);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    // tet size, distance of the tet from the origin, step over size, flatness
    const double kinds[][4] = {{2e-3, 0.2, 0.02, 1.0},  {2e-3, 0.2, 2.0, 1.0},   {1e-2, 0.1, 0.003, 1.0},
                               {2e-3, 0.2, 0.05, 1e-3}, {1e-6, 0.2, 0.1, 1.0},   {1.0, 1000.0, 0.1, 1.0},
                               {1e-3, 0.0, 0.1, 1.0},   {1e-9, 1e-9, 0.5, 1.0},  {1e5, 1e7, 0.3, 1.0},
                               {2e-3, 1e60, 0.5, 1.0},  {2e-3, 0.2, 1e-7, 1.0}};
    for (const auto &k : kinds) {
        long decided = 0, undecided = 0, wrong = 0;
        for (int it = 0; it < 400000; ++it) {
            double v[4][3], o[3];
            for (double &c : o) c = k[1] * (2.0 * u(g) - 1.0);
            for (auto &r : v)
                for (int c = 0; c < 3; ++c) r[c] = o[c] + k[0] * (u(g) - 0.5) * (c == 2 ? k[3] : 1.0);
            const Tet t = make(v);
            // start point in the tet (or, half of the time with an entry face, anywhere near it)
            double w[4], s = 0.0, p0[3], p1[3];
            for (double &x : w) s += x = -std::log(u(g) + 1e-300);
            int enter = -1;
            const int how = int(u(g) * 6);
            if (how == 1) w[int(u(g) * 4)] = 0.0;               // on a face
            if (how == 2) w[0] = w[1] = 0.0;                    // on an edge
            if (how == 3) enter = int(u(g) * 4);                // entered by a crossing
            s = w[0] + w[1] + w[2] + w[3];
            for (int c = 0; c < 3; ++c) p0[c] = (w[0] * v[0][c] + w[1] * v[1][c] + w[2] * v[2][c] + w[3] * v[3][c]) / s;
            if (how == 3)
                for (double &c : p0) c += k[0] * (u(g) - 0.5);
            for (int c = 0; c < 3; ++c) p1[c] = p0[c] + k[0] * k[2] * 2.0 * (u(g) - 0.5) * (c == 2 ? k[3] : 1.0);
            if (how == 4)  // through an edge or a vertex of the tet
                for (int c = 0; c < 3; ++c) p1[c] = p0[c] + 1.5 * (v[1][c] - p0[c]);
            if (how == 5)  // onto a vertex
                for (int c = 0; c < 3; ++c) p1[c] = v[2][c];
            const int a = screen_exit(t.Mf, t.x0, p0, p1, enter), b = exact(t, p0, p1, enter);
            if (a == kScreenUndecided)
                ++undecided;
            else if (a == b)
                ++decided;
            else
                ++wrong;
        }
        std::printf("%ld %ld %ld\n", decided, undecided, wrong);
    }
    return 0;
}
