// Bond detection against the plain double loop over i < j: the same pairs in the same order, for every size,
// critical separation and position the entry point takes (ties along x, coincident points, points at exactly
// the bonding distance, non-finite coordinates).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include <numeric>
#include <utility>
#include <vector>

using Bonds = std::vector<std::pair<int32_t, int32_t>>;
int lg_detect_bonds(const double *x0, int64_t n, double r, double dc, bool cycle_free, Bonds &bonds, bool inclusive);

static Bonds plain(const std::vector<double> &x, int64_t n, double r, double dc, bool cycle_free, bool inclusive) {
    Bonds out;
    std::vector<int64_t> set((size_t)n);
    std::iota(set.begin(), set.end(), 0);
    for (int64_t i = 0; i + 1 < n; ++i)
        for (int64_t j = i + 1; j < n; ++j) {
            const double a = x[3 * i] - x[3 * j], b = x[3 * i + 1] - x[3 * j + 1], c = x[3 * i + 2] - x[3 * j + 2];
            const double g = std::sqrt((a * a + b * b) + c * c) - 2.0 * r;
            if (inclusive ? std::fabs(g) > dc : !(std::fabs(g) < dc)) continue;
            if (cycle_free) {
                if (set[i] == set[j]) continue;
                const int64_t from = set[j], to = set[i];
                for (auto &s : set)
                    if (s == from) s = to;
            }
            out.emplace_back((int32_t)i, (int32_t)j);
        }
    return out;
}

static uint64_t state = 12345;
static double uniform() {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(state >> 11) * 0x1.0p-53;
}

int main() {
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
    const double r = 1.4e-8;
    int bad = 0;
    for (int64_t n : {1, 2, 3, 40, 257, 600})
        for (int shape = 0; shape < 5; ++shape) {
            std::vector<double> x(3 * (size_t)n);
            const double side = 2.0 * r * std::cbrt((double)n);
            for (int64_t i = 0; i < n; ++i)
                for (int c = 0; c < 3; ++c) {
                    const int64_t cell = c == 0 ? i % 7 : c == 1 ? (i / 7) % 7 : i / 49;
                    x[3 * i + c] = shape == 0   ? side * uniform()                            // a dense cloud
                                   : shape == 1 ? 2.0 * r * (double)cell                      // a lattice at contact
                                   : shape == 2 ? 2.0 * r * (double)cell + 1e-12 * r * (uniform() - 0.5)
                                   : shape == 3 ? 1e3 * side + (c == 0 ? 0.0 : side * uniform())  // one plane, far away
                                                : (i % 3 ? side * uniform() : 0.0);           // coincident points
                }
            for (int odd = 0; odd < 3; ++odd) {
                if (odd == 1) x[3 * (n / 2)] = nan;
                if (odd == 2) x[3 * (n / 2)] = -inf;
                for (double dc : {0.0, 1e-10 * r, 0.5 * r, -r, -3.0 * r, 1e3 * r, inf, nan})
                    for (int flags = 0; flags < 4; ++flags) {
                        Bonds got;
                        lg_detect_bonds(x.data(), n, r, dc, flags & 1, got, flags & 2);
                        if (got != plain(x, n, r, dc, flags & 1, flags & 2)) {
                            std::printf("n %lld shape %d odd %d dc %g flags %d differs\n", (long long)n, shape, odd, dc, flags);
                            ++bad;
                        }
                    }
            }
        }
    return bad != 0;
}
