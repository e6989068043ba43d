// Bond detection at the sizes and shapes where its algorithm changes, against a plain double loop over i < j: the
// same pairs in the same order. Then prints the ms that an aggregate, a chain along z, the plane x = 0 and a
// compact cluster of 8192 take.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <numeric>
#include <utility>
#include <vector>

using Bonds = std::vector<std::pair<int32_t, int32_t>>;
int lg_detect_bonds(const double *x0, int64_t n, double r, double dc, bool cycle_free, Bonds &bonds, bool inclusive);
extern "C" int lg_generate_rsa_aggregate(uint64_t seed, int64_t n, double r, double *x);

static int32_t root(std::vector<int32_t> &p, int32_t a) {
    while (p[a] != a) a = p[a] = p[p[a]];
    return a;
}
static Bonds plain(const std::vector<double> &x, int64_t n, double r, double dc, bool cycle_free, bool inclusive) {
    Bonds out;
    std::vector<int32_t> set((size_t)n);
    std::iota(set.begin(), set.end(), 0);
    for (int64_t i = 0; i + 1 < n; ++i)
        for (int64_t j = i + 1; j < n; ++j) {
            const double a = x[3 * i] - x[3 * j], b = x[3 * i + 1] - x[3 * j + 1], c = x[3 * i + 2] - x[3 * j + 2];
            const double g = std::sqrt((a * a + b * b) + c * c) - 2.0 * r;
            if (inclusive ? std::fabs(g) > dc : !(std::fabs(g) < dc)) continue;
            if (cycle_free) {
                const int32_t ra = root(set, (int32_t)i), rb = root(set, (int32_t)j);
                if (ra == rb) continue;
                set[rb] = ra;
            }
            out.emplace_back((int32_t)i, (int32_t)j);
        }
    return out;
}

static uint64_t state = 777;
static double uniform() {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(state >> 11) * 0x1.0p-53;
}

static const double r = 1.4e-8;
static std::vector<double> shape_of(int shape, int64_t n) {
    std::vector<double> x(3 * (size_t)n);
    const double side = 2.0 * r * std::cbrt((double)n), square = 2.0 * r * std::sqrt((double)n);
    if (shape == 0) lg_generate_rsa_aggregate(5, n, r, x.data());
    for (int64_t i = 0; i < n && shape; ++i)
        for (int c = 0; c < 3; ++c)
            x[3 * i + c] = shape == 1   ? (c == 2 ? 2.0 * r * (double)i : 0.0)  // a chain along z
                           : shape == 2 ? (c == 0 ? 0.0 : square * uniform())   // the plane x = 0
                           : shape == 3 ? side * uniform()                      // a cloud
                                        : 3.0 * r * uniform();                  // a compact cluster
    return x;
}

int main() {
    int bad = 0;
    for (int64_t n : {2047, 2048, 2049, 8192, 8193})
        for (int shape = 0; shape < 5; ++shape) {
            if (shape == 4 && n > 2049) continue;  // (most of its pairs bond)
            const std::vector<double> x = shape_of(shape, n);
            for (double dc : {1e-10 * r, 0.05 * r})
                for (int flags = 0; flags < 4; flags += n > 2049 ? 3 : 1) {
                    Bonds got;
                    lg_detect_bonds(x.data(), n, r, dc, flags & 1, got, flags & 2);
                    if (got != plain(x, n, r, dc, flags & 1, flags & 2)) {
                        std::printf("n %lld shape %d dc %g flags %d differs\n", (long long)n, shape, dc, flags);
                        ++bad;
                    }
                }
        }
    if (bad) return 1;
    for (int shape : {0, 1, 2, 4}) {
        const int64_t n = 8192;
        std::vector<double> x = shape_of(shape, n);
        double best = 1e9;
        for (int k = 0; k < 7; ++k) {
            Bonds got;
            const auto t0 = std::chrono::steady_clock::now();
            lg_detect_bonds(x.data(), n, r, 1e-10 * r, true, got, false);
            best = std::min(best, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
        }
        std::printf("%.4f\n", best);
    }
    return 0;
}
