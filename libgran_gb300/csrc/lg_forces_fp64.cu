// lg_forces_fp64.cu -- FP64 row-group force evaluation and integration kernels (sm_103a).
//
// Compiled with --fmad=false: a thread that walks its row in ascending j evaluates every pair with
// the same operations, in the same order, as libgran's functors evaluated sequentially on a CPU
// (see lg_common.cuh). One "row group" of T consecutive lanes (T in {1, 2, 4, 8, 16, 32}) owns one
// particle i: lane l handles slots k = l, l + T, ... of row i, and the group then combines its T
// partial sums with a fixed xor-butterfly. T = 1 reproduces the sequential sum bit for bit; larger
// T spreads short, FP64-heavy rows (all-pairs mode on a few hundred particles) over more of the
// GPU's FP64 units. No floating-point atomics are used anywhere: every per-particle sum is owned
// by one row group, so results are deterministic run to run.
#include "lg_compact.cuh"
#include "lg_kernels.h"
#include "lg_pair_fp64.cuh"

namespace lg {

// ------------------------------------------------------------------------------------------------
// Kick + drift (first half of the rotational velocity-Verlet step):
//   v += a*(dt/2); w += al*(dt/2); x += v*dt; th += w*dt
// ------------------------------------------------------------------------------------------------
__global__ void kick_drift_fp64(int64_t n, dbl4 *__restrict__ x, dbl4 *__restrict__ v,
                                dbl4 *__restrict__ th, dbl4 *__restrict__ w, const dbl4 *__restrict__ a,
                                const dbl4 *__restrict__ al, double dt, double hdt, BondView BV,
                                const uint8_t *__restrict__ hold) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t h = hold_of(hold, i);
    d3 vi = kick_unless(ld4(v, i), hdt, ld4(a, i), h & LG_HOLD_V);
    d3 wi = kick_unless(ld4(w, i), hdt, ld4(al, i), h & LG_HOLD_OMEGA);
    st4(v, i, vi);
    st4(w, i, wi);
    drift_one(n, i, x, th, vi, wi, dt, BV, h);
}

// Body force LG_BODY_CENTRAL (central_attraction_functor, Custom-unary-force-model.md:108-118):
// a = k_a / mass * (centre - x_i), alpha = 0; kam = k_a / mass (formed on the host, as the
// functor forms it); one centre per system.
__global__ void body_central(int64_t n, const dbl4 *__restrict__ x, const int32_t *__restrict__ agg,
                             const double *__restrict__ centre, double kam, dbl4 *__restrict__ ea,
                             dbl4 *__restrict__ eal) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t q = agg ? (int64_t)agg[i] : 0;
    const d3 c = mk3(centre[3 * q], centre[3 * q + 1], centre[3 * q + 2]);
    st4(ea, i, scl(kam, sub(c, ld4(x, i))));
    st4(eal, i, zero3());
}

// ------------------------------------------------------------------------------------------------
// Pair force kernel
// ------------------------------------------------------------------------------------------------
template <int T>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int T, bool VERLET>
__global__ void __launch_bounds__(256) forces_fp64(Params P, StateView S, PairView PV, BondView BV, double hdt,
                                                   double dt, int move_facets) {
    const int64_t n = P.n;
    const int64_t gid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t i = gid / T;
    const int lane = (int)(gid % T);
    const bool active = i < n;

    if (move_facets && gid == 0) {
        for (int f = 0; f < P.n_facets; ++f)
            for (int q = 0; q < 9; ++q) S.facet_vert_next[9 * f + q] = S.facet_vert[9 * f + q] + P.facets[f].v[q % 3] * dt;
    }

    d3 acc = zero3(), accw = zero3();
    d3 xi_ = zero3(), vi = zero3(), wi = zero3();
    if (active) {
        xi_ = ld4(S.x, i);
        vi = ld4(S.v, i);
        wi = ld4(S.w, i);
        const int64_t len = VERLET ? (int64_t)PV.row_len[i] : n - 1;
        const int64_t stride = n;  // slot k of row i lives at k * n + i
        for (int64_t k = lane; k < len; k += T) {
            const int64_t e = k * stride + i;
            const int64_t j = VERLET ? (int64_t)PV.nbr[e] : (k < i ? k : k + 1);
            d3 pa, pal;
            slot_pair_fp64(P, S, PV, BV, n, i, e, j, xi_, vi, wi, pa, pal);
            acc = add(acc, pa);
            accw = add(accw, pal);
        }
    }
    if (T > 1) {
        acc.x = group_sum<T>(acc.x);
        acc.y = group_sum<T>(acc.y);
        acc.z = group_sum<T>(acc.z);
        accw.x = group_sum<T>(accw.x);
        accw.y = group_sum<T>(accw.y);
        accw.z = group_sum<T>(accw.z);
    }
    if (!active || lane != 0) return;
    compact::finish_row(P, S, i, n, acc, accw, vi, wi, hdt);
}

// ------------------------------------------------------------------------------------------------
// Host-side launchers
// ------------------------------------------------------------------------------------------------
template <int T, bool VERLET>
static void launch_forces_t(const Params &P, const StateView &S, const PairView &PV, const BondView &BV, double hdt,
                            double dt, int move_facets, cudaStream_t st) {
    const int threads = 256;
    const int64_t total = P.n * T;
    const int64_t blocks = (total + threads - 1) / threads;
    forces_fp64<T, VERLET><<<(unsigned)(blocks > 0 ? blocks : 1), threads, 0, st>>>(P, S, PV, BV, hdt, dt, move_facets);
}

void launch_forces_fp64(int T, const Params &P, const StateView &S, const PairView &PV, const BondView &BV, double hdt,
                        double dt, int move_facets, cudaStream_t st) {
    const bool ver = P.pairs == LG_PAIRS_VERLET;
#define LG_CASE(TT)                                                                \
    case TT:                                                                       \
        if (ver)                                                                   \
            launch_forces_t<TT, true>(P, S, PV, BV, hdt, dt, move_facets, st);     \
        else                                                                       \
            launch_forces_t<TT, false>(P, S, PV, BV, hdt, dt, move_facets, st);    \
        break;
    switch (T) {
        LG_CASE(1)
        LG_CASE(2)
        LG_CASE(4)
        LG_CASE(8)
        LG_CASE(16)
        LG_CASE(32)
        default:
            launch_forces_t<1, false>(P, S, PV, BV, hdt, dt, move_facets, st);
    }
#undef LG_CASE
}

void launch_body_central(int64_t n, const dbl4 *x, const int32_t *agg, const double *centre, double kam, dbl4 *ea,
                         dbl4 *eal, cudaStream_t st) {
    const int threads = 64;
    const int64_t blocks = (n + threads - 1) / threads;
    if (blocks == 0) return;
    body_central<<<(unsigned)blocks, threads, 0, st>>>(n, x, agg, centre, kam, ea, eal);
}

void launch_kick_drift_fp64(int64_t n, dbl4 *x, dbl4 *v, dbl4 *th, dbl4 *w, const dbl4 *a,
                            const dbl4 *al, double dt, double hdt, const BondView &BV, const uint8_t *hold,
                            cudaStream_t st) {
    const int threads = 64;  // small blocks: all SMs get work at moderate n
    int64_t blocks = (n + threads - 1) / threads;
    if (blocks == 0) return;
    kick_drift_fp64<<<(unsigned)blocks, threads, 0, st>>>(n, x, v, th, w, a, al, dt, hdt, BV, hold);
}

}  // namespace lg
