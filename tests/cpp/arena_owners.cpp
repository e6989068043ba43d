// A serving slot emptied between two list builds: until the next build no owned slot or candidate of its rows is
// left for the pair kernels to walk, the other slot's are all there, and its occupant goes on as it would alone.
// Prints the owners per slot before the clear, after it, and whether the other occupant's state is the lone run's.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "lg_engine_internal.h"

#define OK(call)                                                      \
    do {                                                              \
        if ((call) != LG_OK) {                                        \
            std::printf("%s: %s\n", #call, lg_last_error());          \
            return 1;                                                 \
        }                                                             \
    } while (0)

// owned entries of the rows [b, e): blocks of `rb` rows, a slot's capacity being a multiple of it
static int64_t owners(lg_system *s, int64_t rb, int64_t b, int64_t e) {
    std::vector<int32_t> own((size_t)((s->P.n + rb - 1) / rb));
    cudaStreamSynchronize(s->stream);
    cudaMemcpy(own.data(), s->own_n, sizeof(int32_t) * own.size(), cudaMemcpyDeviceToHost);
    int64_t sum = 0;
    for (int64_t q = b / rb; q < e / rb; ++q) sum += own[(size_t)q];
    return sum;
}

int main(int argc, char **argv) {
    const bool mixed = argc > 1 && !std::strcmp(argv[1], "mixed");
    const double r = 1.4e-8, m = 1.95e-20, I = 0.4 * m * r * r, dt = 1.4e-14;
    lg_system_desc d{};
    d.precision = mixed ? LG_PRECISION_MIXED : LG_PRECISION_FP64;
    d.binary_model = LG_BINARY_SINTER;
    d.hamaker_model = LG_HAMAKER_LIMITED;
    d.pairs = LG_PAIRS_VERLET;
    d.r_verlet = (mixed ? 4.1 : 4.5) * r;  // (mixed: candidates near contact, which are evaluated once per pair)
    d.max_neighbors = 96;
    d.contact = {1e4, 3e-9, 5e3, 2e-9, 1.0, 1.0, 5e3, 2e-9, 1.0, 1.0, 5e3, 2e-9, 1.0, 1.0, r, m, I, dt};
    d.sinter = {1e4, 3e-9, 5e3, 2e-9, 5e3, 2e-9, 5e3, 2e-9, r, m, I, dt, 1e-9};
    d.hamaker = {1e-19, 4e-10, 4.0 * r, r, m};
    const int64_t n = 384, caps[2] = {512, 512};
    std::vector<double> x(3 * n), v(3 * n), zero(3 * n, 0.0);
    OK(lg_generate_rsa_aggregate(11, n, r, x.data()));
    OK(lg_generate_velocities(11, n, 0.1, v.data()));
    d.n_part = n;
    lg_system *arena = nullptr, *stage[2], *lone = nullptr;
    OK(lg_arena_create(&d, 2, caps, 0, &arena));
    d.n_part = n;
    for (int q = 0; q < 2; ++q) {
        OK(lg_create_staged(&d, x.data(), v.data(), 0, &stage[q]));
        OK(lg_arena_import(arena, q, stage[q], x.data()));
        OK(lg_destroy(stage[q]));
    }
    d.force_kernel = LG_FORCE_KERNEL_COMPACT;
    OK(lg_create(&d, x.data(), v.data(), zero.data(), zero.data(), nullptr, nullptr, 0, 0, &lone));
    const int64_t rb = mixed ? lg::near_block_rows(1024) : lg::pair_block_rows(1024);
    OK(lg_step(arena, dt, 27, 20));
    const int64_t b0 = owners(arena, rb, 0, 512), b1 = owners(arena, rb, 512, 1024);
    OK(lg_arena_clear(arena, 0));
    OK(lg_step(arena, dt, 5, 20));
    const int64_t a0 = owners(arena, rb, 0, 512), a1 = owners(arena, rb, 512, 1024);
    OK(lg_step(arena, dt, 31, 20));
    OK(lg_step(lone, dt, 27, 20));
    OK(lg_step(lone, dt, 5, 20));
    OK(lg_step(lone, dt, 31, 20));
    std::vector<double> xa(3 * n), xl(3 * n);
    OK(lg_arena_read(arena, 1, n, xa.data(), nullptr, nullptr, nullptr));
    OK(lg_get(lone, LG_FIELD_X, xl.data()));
    int32_t errs = 0;
    OK(lg_get_device_errors(arena, &errs));
    std::printf("%lld %lld %lld %lld %d %d\n", (long long)b0, (long long)b1, (long long)a0, (long long)a1,
                std::memcmp(xa.data(), xl.data(), sizeof(double) * 3 * n) == 0, errs);
    OK(lg_destroy(arena));
    OK(lg_destroy(lone));
    return 0;
}
