// lg_forces_pairs.cu -- FP64 force evaluation over unordered pairs (sm_103a); compiled with --fmad=false.
// Two instances: the reference's arithmetic operation for operation (bit-identical to the sequential
// evaluation), and FAST (LG_FORCE_KERNEL_FP64_FAST), which multiplies by one reciprocal where libgran
// divides a vector by a scalar and evaluates the Hamaker bracket over one common denominator (per-step
// forces within 1e-12 of the reference's); both decide contact with the reference's exact overlap.
//
// What bounds it: GB300 issues one FP64 warp instruction per SM sub-partition about every 64 cycles,
// however many lanes are active, so the time is the number of FP64 warp instructions on the busiest
// sub-partition. Three things keep that number low:
//   * every unordered pair is evaluated once. The Hamaker term of (j, i) is the exact negative of that
//     of (i, j): each of its operations only changes sign with the separation, and rounding to nearest
//     is symmetric. Contact and bond values are not (their relative velocity adds the two rotation
//     terms in row order), so those run for both orders;
//   * full warps: pairs are taken from a compact list of owned slots (built with the Verlet rows; all
//     pairs: by index), and the contact and bond slots found in a block are queued in shared memory and
//     evaluated 32 at a time;
//   * small blocks spread over all SMs, with one warp of each block for the queue, so that a small
//     system's long contact evaluations (about 300 dependent FP64 instructions) run beside its Hamaker
//     terms.
// Each slot's value (binary + Hamaker, added as the reference's container adds them) goes to a record in
// device memory; pair_fold then adds each row's records in ascending slot order, exactly as the
// sequential row loop does, six lanes per row, one component each (a row's sum is one dependent chain
// per component), and goes on to the half kick and, inside a run of steps, the next step's kick and
// drift of that component. Every slot is written by one thread and every sum has a fixed order, so
// results do not depend on scheduling.
#include <algorithm>

#include "lg_compact.cuh"
#include "lg_kernels.h"
#include "lg_pair_fp64.cuh"

namespace lg {

namespace {

constexpr uint32_t kNoRev = 255u;  // the partner's row does not list the slot's row (a truncated row)
constexpr int kPairBlock = 128;    // threads per block of pair_hamaker (fewer for small systems)
constexpr int kContactBlock = 64;

}  // namespace

// The owned slots of each block of `rb` rows: of the two slots of a pair (i, j) the one in row i when
// i < j and i + j is odd, or i > j and i + j is even (so that every row owns about half of its slots);
// a slot whose partner's row does not list it is always owned. Entry: partner, local row, slot and the
// slot of i in the partner's (ascending) row, found by bisection.
__global__ void __launch_bounds__(128) pair_owners(int64_t n, PairView PV, PairScratch R) {
    __shared__ int32_t cnt;
    __shared__ int32_t lmax;
    const int tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * R.rb;
    if (tid == 0) cnt = lmax = 0;
    __syncthreads();
    if (tid < R.rb && row0 + tid < n) atomicMax(&lmax, PV.row_len[row0 + tid]);
    __syncthreads();
    uint2 *own = R.own + row0 * PV.cap;
    const int total = R.rb * lmax;
    for (int q = tid; q < total; q += blockDim.x) {
        const int r = q % R.rb, k = q / R.rb;
        const int64_t i = row0 + r;
        if (i >= n || k >= PV.row_len[i]) continue;
        const int32_t j = PV.nbr[(int64_t)k * n + i];
        const int32_t lj = PV.row_len[j];
        int lo = 0, hi = lj;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (PV.nbr[(int64_t)mid * n + j] < (int32_t)i) lo = mid + 1;
            else hi = mid;
        }
        const uint32_t rev = lo < lj && PV.nbr[(int64_t)lo * n + j] == (int32_t)i ? (uint32_t)lo : kNoRev;
        const bool mine = rev == kNoRev || (((i + j) & 1) ? i < j : i > j);
        if (mine) own[atomicAdd(&cnt, 1)] = make_uint2((uint32_t)j, (uint32_t)r | ((uint32_t)k << 8) | (rev << 16));
    }
    __syncthreads();
    if (tid == 0) R.own_n[blockIdx.x] = cnt;
}

// Classifies the pairs of a block, one per lane, and evaluates their Hamaker terms (0 where there is
// none); pairs that are bonded, within contact reach or have springs to reset go to the contact queue,
// both orders. VERLET: block b takes the owned slots of its rows; all pairs: pairs [b * per, (b + 1) *
// per) of the enumeration (i, i + d mod n), d ascending.
template <bool VERLET, bool FAST>
__global__ void __launch_bounds__(kPairBlock) pair_hamaker(Params P, StateView S, PairView PV, PairScratch R,
                                                           int32_t per) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t n = P.n;
    const int bm = P.binary_model, hm = P.hamaker_model;
    int32_t count, p0 = 0;
    const uint2 *own = nullptr;
    if (VERLET) {
        count = R.own_n[blockIdx.x];
        own = R.own + (int64_t)blockIdx.x * R.rb * PV.cap;
    } else {
        p0 = blockIdx.x * per;
        const int32_t total = (int32_t)(n * (n - 1) / 2);
        count = total - p0 < per ? total - p0 : per;
    }
    for (int32_t c0 = tid - lane; c0 < count; c0 += blockDim.x) {
        const int32_t c = c0 + lane;
        int64_t i = 0, j = 0, e = 0, e2 = -1;
        int32_t k = 0, k2 = 0;
        d3 r = zero3();
        double d2 = 0.0;
        const bool live = c < count;
        bool touch = false;
        if (live) {
            if (VERLET) {
                const uint2 o = own[c];
                j = o.x;
                i = (int64_t)blockIdx.x * R.rb + (o.y & 0xffu);
                k = (int32_t)((o.y >> 8) & 0xffu);
                k2 = (int32_t)(o.y >> 16);
            } else {
                const uint32_t p = (uint32_t)(p0 + c), un = (uint32_t)n, d = p / un + 1u;
                i = p - (d - 1u) * un;
                j = i + d;
                if (j >= n) j -= n;
                k = (int32_t)(j < i ? j : j - 1);
                k2 = (int32_t)(i < j ? i : i - 1);
            }
            const bool both = !VERLET || k2 != (int32_t)kNoRev;
            e = (int64_t)k * n + i;
            if (both) e2 = (int64_t)k2 * n + j;
            uint32_t fl = 0;
            if (bm != LG_BINARY_NONE) {
                fl = PV.flags[e];
                if (both) fl |= PV.flags[e2];
            }
            r = sub(ld4(S.x, j), ld4(S.x, i));
            d2 = sqn(r);
            touch = bm != LG_BINARY_NONE && ((fl & (kBonded | kXiLive)) || !above(d2, P.contact_skip_d2));
        }
        if (bm != LG_BINARY_NONE) {  // queue places for the warp's contact slots with one atomic
            const uint32_t b1 = __ballot_sync(0xffffffffu, touch), b2 = __ballot_sync(0xffffffffu, touch && e2 >= 0);
            if (b1) {
                int q = 0;
                if (lane == 0) q = atomicAdd(R.q_n, __popc(b1) + __popc(b2));
                const uint32_t lt = (1u << lane) - 1u;
                q = __shfl_sync(0xffffffffu, q, 0) + __popc(b1 & lt) + __popc(b2 & lt);
                if (touch) {
                    R.q_i[q] = (int32_t)i;
                    R.q_k[q] = k;
                    if (e2 >= 0) {
                        R.q_i[q + 1] = (int32_t)j;
                        R.q_k[q + 1] = k2;
                    }
                }
            }
        }
        if (!live) continue;
        d3 a = zero3();
        if (hm != LG_HAMAKER_NONE && !(hm == LG_HAMAKER_LIMITED && above(d2, P.hamaker_skip_d2))) {
            const double rn = droot(d2);
            if (!(hm == LG_HAMAKER_LIMITED && above(rn, P.hamaker.r_cutoff)))
                a = hamaker_accel_n<FAST>(hm, P.hamaker, r, rn);
        }
        st4(R.rec, e, a);
        if (e2 >= 0) st4(R.rec, e2, neg(a));
    }
}

// Contact and bond values of the queued slots, one per lane, added to the slot's Hamaker term (the
// reference's container adds binary + Hamaker); w = 1 marks a record with a torque part.
template <bool VERLET, bool FAST, bool CONNECTORS>
__global__ void __launch_bounds__(kContactBlock) pair_contacts(Params P, StateView S, PairView PV, BondView BV,
                                                               PairScratch R) {
    const int64_t n = P.n;
    const int32_t total = *R.q_n;
    const bool ham = P.hamaker_model != LG_HAMAKER_NONE;
    for (int32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
        const int64_t i = R.q_i[q], k = R.q_k[q], e = k * n + i;
        const int64_t j = VERLET ? (int64_t)PV.nbr[e] : (k < i ? k : k + 1);
        d3 pb, pbl, pa, pal;
        slot_binary_fp64<FAST, CONNECTORS>(P, S, PV, BV, n, i, e, j, ld4(S.x, i), ld4(S.v, i), ld4(S.w, i), pb, pbl);
        combine_pair_fp64(true, ham, pb, pbl, ld4(R.rec, e), pa, pal);
        R.rec[e] = make_double4_32a(pa.x, pa.y, pa.z, 1.0);
        st4(R.tq, e, pal);
    }
}

constexpr int kFoldBlock = 32;
constexpr int kFoldRows = 5;    // rows per warp of the fold (six lanes each)
constexpr int kFoldAhead = 8;   // slots whose pair terms a lane of the fold has in flight

// Lane 6 r + c of a warp sums component c (force x, y, z, torque x, y, z) of the warp's row r in slot
// order, the next kFoldAhead slots' loads in flight during the additions of the current ones. Records
// without a binary part carry no torque (and tag 0); a zero added to a sum that started at +0 leaves
// its bits alone, so torque lanes skip those.
template <bool VERLET, bool FACETS>
__global__ void __launch_bounds__(kFoldBlock) pair_fold(Params P, StateView S, PairView PV, BondView BV, PairScratch R,
                                                        double hdt, double dt, int move_facets, int kick) {
    const int64_t n = P.n;
    if (move_facets && blockIdx.x == 0 && threadIdx.x == 0) compact::move_facets(P, S, dt);
    const int lane = threadIdx.x & 31;
    const int r = lane / 6, c = lane % 6;
    const int64_t i = (int64_t)blockIdx.x * kFoldRows + r;
    const bool mine = r < kFoldRows && i < n;
    const bool torque = c >= 3;
    double sum = 0.0, vel = 0.0;
    uint32_t h = 0;
    if (mine) {
        const int64_t len = VERLET ? (int64_t)PV.row_len[i] : n - 1;
        const double *vs = reinterpret_cast<const double *>(torque ? S.w : S.v);
        vel = vs[4 * i + (torque ? c - 3 : c)];
        h = hold_of(P.hold, i);
        const double *col = reinterpret_cast<const double *>(R.rec) + 4 * i + (torque ? 3 : c);
        const double *tq = reinterpret_cast<const double *>(R.tq) + 4 * i + (c - 3);
        const int64_t pitch = 4 * n;
        double t[kFoldAhead], u[kFoldAhead];
#pragma unroll
        for (int q = 0; q < kFoldAhead; ++q) t[q] = q < len ? col[q * pitch] : 0.0;
        for (int64_t k = 0; k < len; k += kFoldAhead) {
#pragma unroll
            for (int q = 0; q < kFoldAhead; ++q) {
                const int64_t kk = k + kFoldAhead + q;
                u[q] = kk < len ? col[kk * pitch] : 0.0;
            }
            if (torque) {
#pragma unroll
                for (int q = 0; q < kFoldAhead; ++q)
                    if (__double_as_longlong(t[q]) != 0) t[q] = tq[(k + q) * pitch];
            }
#pragma unroll
            for (int q = 0; q < kFoldAhead; ++q) sum += t[q];
#pragma unroll
            for (int q = 0; q < kFoldAhead; ++q) t[q] = u[q];
        }
    }
    if (FACETS) {  // unary terms of the whole row, on the row's first lane
        double f[6], w[6];
        const int src = r < kFoldRows ? 6 * r : 0;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            f[q] = __shfl_sync(0xffffffffu, sum, src + q);
            w[q] = __shfl_sync(0xffffffffu, vel, src + q);
        }
        if (mine && c == 0) {
            d3 ua, ual;
            if (compact::unary_terms(P, S, i, n, mk3(w[0], w[1], w[2]), mk3(w[3], w[4], w[5]), ua, ual)) {
                f[0] += ua.x;
                f[1] += ua.y;
                f[2] += ua.z;
                f[3] += ual.x;
                f[4] += ual.y;
                f[5] += ual.z;
            }
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const double g = __shfl_sync(0xffffffffu, f[q], src);
            if (q == c) sum = g;
        }
    }
    const int cc = torque ? c - 3 : c;
    const bool hv = h & (torque ? LG_HOLD_OMEGA : LG_HOLD_V);
    double v1 = vel;
    if (blockIdx.x == 0 && lane == 31) *R.q_n = 0;  // the next evaluation's queue
    if (mine) {
        reinterpret_cast<double *>(torque ? S.al : S.a)[4 * i + cc] = sum;
        if (!isfinite(sum)) set_error(S.err, LG_DEVERR_NONFINITE);
        if (!hv) v1 = vel + hdt * sum;
        if (kick && !hv) v1 = v1 + hdt * sum;  // the next step's opening half kick
        reinterpret_cast<double *>(torque ? S.w_out : S.v_out)[4 * i + cc] = v1;
    }
    if (!kick) return;
    if (!BV.cn) {  // the next step's drift of this component
        if (mine && !(h & (torque ? LG_HOLD_THETA : LG_HOLD_X))) {
            double *p = reinterpret_cast<double *>(torque ? S.th : S.x) + 4 * i + cc;
            *p = *p + dt * v1;
        }
        return;
    }
    // with connectors the drift needs the whole particle
    double f[6];
    const int src = r < kFoldRows ? 6 * r : 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) f[q] = __shfl_sync(0xffffffffu, v1, src + q);
    if (mine && c == 0) drift_one(n, i, S.x, S.th, mk3(f[0], f[1], f[2]), mk3(f[3], f[4], f[5]), dt, BV, h);
}

// Rows per block of owned slots: enough blocks for every SM, and as many rows as that allows (fuller
// contact batches).
int32_t pair_block_rows(int64_t n) { return n >= 16384 ? 32 : n >= 5000 ? 16 : n >= 2500 ? 8 : 4; }

void launch_pair_owners(int64_t n, const PairView &PV, const PairScratch &R, cudaStream_t st) {
    const unsigned blocks = (unsigned)((n + R.rb - 1) / R.rb);
    if (blocks) pair_owners<<<blocks, 128, 0, st>>>(n, PV, R);
}

namespace {
template <bool FAST>
int launch_pairs(const Params &P, const StateView &S, const PairView &PV, const BondView &BV, const PairScratch &R,
                 double hdt, double dt, int move_facets, bool kick, cudaStream_t st) {
    const int64_t n = P.n;
    const bool verlet = P.pairs == LG_PAIRS_VERLET;
    int kernels = 1;
    if (n > 1) {
        unsigned blocks, threads = kPairBlock;
        int32_t per = 0;
        if (verlet) {
            blocks = (unsigned)((n + R.rb - 1) / R.rb);
            if (R.rb <= 8) threads = 64;
            pair_hamaker<true, FAST><<<blocks, threads, 0, st>>>(P, S, PV, R, per);
        } else {  // 64 pairs per block while that fills the GPU about twice, then up to four rounds of 128
            const int64_t total = n * (n - 1) / 2;
            if (total <= 64 * 1216) {
                per = threads = 64;
            } else {
                per = 128;
                while (per < 512 && total > (int64_t)per * 1216) per += 128;
            }
            blocks = (unsigned)((total + per - 1) / per);
            pair_hamaker<false, FAST><<<blocks, threads, 0, st>>>(P, S, PV, R, per);
        }
        ++kernels;
    }
    if (n > 1 && P.binary_model != LG_BINARY_NONE) {
        const int64_t slots = (verlet ? std::min<int64_t>(PV.cap, 16) : std::min<int64_t>(n - 1, 16)) * n;
        const unsigned blocks = (unsigned)std::min<int64_t>((slots + kContactBlock - 1) / kContactBlock, 152 * 8);
        if (BV.cn) {
            if (verlet) pair_contacts<true, FAST, true><<<blocks, kContactBlock, 0, st>>>(P, S, PV, BV, R);
            else pair_contacts<false, FAST, true><<<blocks, kContactBlock, 0, st>>>(P, S, PV, BV, R);
        } else {
            if (verlet) pair_contacts<true, FAST, false><<<blocks, kContactBlock, 0, st>>>(P, S, PV, BV, R);
            else pair_contacts<false, FAST, false><<<blocks, kContactBlock, 0, st>>>(P, S, PV, BV, R);
        }
        ++kernels;
    }
    const unsigned fb = (unsigned)((n + kFoldRows - 1) / kFoldRows);  // one warp per kFoldRows rows
    const int kk = kick ? 1 : 0;
    const bool unary = P.n_facets > 0 || P.ext_a;
    if (verlet) {
        if (unary) pair_fold<true, true><<<fb, kFoldBlock, 0, st>>>(P, S, PV, BV, R, hdt, dt, move_facets, kk);
        else pair_fold<true, false><<<fb, kFoldBlock, 0, st>>>(P, S, PV, BV, R, hdt, dt, move_facets, kk);
    } else {
        if (unary) pair_fold<false, true><<<fb, kFoldBlock, 0, st>>>(P, S, PV, BV, R, hdt, dt, move_facets, kk);
        else pair_fold<false, false><<<fb, kFoldBlock, 0, st>>>(P, S, PV, BV, R, hdt, dt, move_facets, kk);
    }
    return kernels;
}
}  // namespace

int launch_forces_pairs_fp64(const Params &P, const StateView &S, const PairView &PV, const BondView &BV,
                             const PairScratch &R, double hdt, double dt, int move_facets, bool kick, bool fast,
                             cudaStream_t st) {
    return fast ? launch_pairs<true>(P, S, PV, BV, R, hdt, dt, move_facets, kick, st)
                : launch_pairs<false>(P, S, PV, BV, R, hdt, dt, move_facets, kick, st);
}

}  // namespace lg
