// The autotuner times shapes of the persistent kernel that the graphs' key does not tell apart: a handle that it
// leaves holds no graph of another shape. Prints the graphs held after the tuning, and after a run with the pick the
// launches of an eager period and of a replayed one (a period's launches depend on the shape).
#include <cstdio>
#include <vector>

#include "lg_engine_internal.h"

int main() {
    const double r = 1.4e-8, m = 1.95e-20, I = 0.4 * m * r * r, dt = 1.4e-14;
    lg_system_desc d{};
    d.precision = LG_PRECISION_MIXED;
    d.binary_model = LG_BINARY_CONTACT;
    d.hamaker_model = LG_HAMAKER_LIMITED;
    d.pairs = LG_PAIRS_VERLET;
    d.r_verlet = 4.5 * r;
    d.max_neighbors = 96;
    d.contact = {1e4, 3e-9, 5e3, 2e-9, 1.0, 1.0, 5e3, 2e-9, 1.0, 1.0, 5e3, 2e-9, 1.0, 1.0, r, m, I, dt};
    d.hamaker = {1e-19, 4e-10, 4.0 * r, r, m};
    const int64_t n = 700;
    d.n_part = n;
    std::vector<double> x(3 * n), zero(3 * n, 0.0);
    lg_generate_rsa_aggregate(11, n, r, x.data());
    lg_system *s = nullptr;
    int32_t kernel = 0, T = 0;
    if (lg_create(&d, x.data(), zero.data(), zero.data(), zero.data(), nullptr, nullptr, 0, 0, &s) != LG_OK ||
        lg_autotune(s, dt, 40, 20, &kernel, &T, 0) != LG_OK) {
        std::printf("%s\n", lg_last_error());
        return 1;
    }
    const int held = (int)s->graphs.size();
    s->kernel = LG_FORCE_KERNEL_PERSISTENT;
    s->step_assign = 2;  // two launches a step
    int64_t a = 0, b = 0, c = 0;
    lg_get_launch_count(s, &a);
    s->use_graphs = false;
    lg_step(s, dt, 20, 20);
    lg_get_launch_count(s, &b);
    s->use_graphs = true;
    lg_step(s, dt, 20, 20);
    lg_get_launch_count(s, &c);
    std::printf("%d %lld %lld\n", held, (long long)(b - a), (long long)(c - b));
    lg_destroy(s);
    return 0;
}
