// What a staged serving handle takes from the pool: for each precision, functor set and size, the bytes of its
// first chunk, the bytes of it that its buffers use, the number of chunks, and the estimate the server charges.
#include <cstdio>
#include <vector>

#include "lg_engine_internal.h"

int main() {
    const double r = 1.4e-8, m = 1.95e-20, I = 0.4 * m * r * r, dt = 1.4e-14;
    for (int precision : {LG_PRECISION_FP64, LG_PRECISION_MIXED})
        for (int model : {LG_BINARY_CONTACT, LG_BINARY_SINTER})
            for (int64_t n : {1, 2, 64, 300, 1024, 4096}) {
                lg_system_desc d{};
                d.precision = precision;
                d.binary_model = model;
                d.hamaker_model = LG_HAMAKER_LIMITED;
                d.pairs = LG_PAIRS_VERLET;
                d.r_verlet = 4.5 * r;
                d.max_neighbors = 96;
                d.n_part = n;
                d.contact = {1e4, 3e-9, 5e3, 2e-9, 1.0, 1.0, 5e3, 2e-9, 1.0, 1.0, 5e3, 2e-9, 1.0, 1.0, r, m, I, dt};
                d.sinter = {1e4, 3e-9, 5e3, 2e-9, 5e3, 2e-9, 5e3, 2e-9, r, m, I, dt, 1e-9};
                d.hamaker = {1e-19, 4e-10, 4.0 * r, r, m};
                std::vector<double> x(3 * n), v(3 * n, 0.0);
                lg_generate_rsa_aggregate(11, n, r, x.data());
                const int64_t chunk = (int64_t)lg_handle_bytes(&d, n), charged = lg_estimate_device_bytes(&d, n);
                lg_system *s = nullptr;
                if (lg_create_staged(&d, x.data(), v.data(), 0, &s) != LG_OK) {
                    std::printf("lg_create_staged: %s\n", lg_last_error());
                    return 1;
                }
                std::printf("%d %d %lld %lld %lld %d %lld\n", precision, model, (long long)n, (long long)chunk,
                            (long long)(chunk - (int64_t)s->slab_left), (int)s->chunks.size(), (long long)charged);
                lg_destroy(s);
            }
    return 0;
}
