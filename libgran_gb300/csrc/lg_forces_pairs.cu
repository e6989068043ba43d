// lg_forces_pairs.cu -- FP64 force evaluation over unordered pairs (sm_103a); compiled with --fmad=false.
// Two instances: the reference's arithmetic operation for operation (bit-identical to the sequential
// evaluation), and FAST (LG_FORCE_KERNEL_FP64_FAST), which multiplies by one reciprocal where libgran
// divides a vector by a scalar and evaluates the Hamaker bracket over one common denominator (per-step
// forces within 1e-12 of the reference's); both decide contact with the reference's exact overlap.
//
// What bounds it: the FP64 unit takes one warp instruction per SM about every 16 cycles (one per
// sub-partition every 64), however many lanes are active, and a dependent one follows after about 70; so
// the time is the number of FP64 warp instructions, and for a small system one pair's chain of them.
//   pair_hamaker   every unordered pair once. The Hamaker term of (j, i) is the exact negative of that of
//                  (i, j): each of its operations only changes sign with the separation, and rounding to
//                  nearest is symmetric. Pairs come from a compact list of owned slots (built with the
//                  Verlet rows; all pairs: by index); those in range are collected per block and evaluated
//                  with full warps. Comparisons run on the integer pipe.
//   pair_contacts  contact and bond values (about 300 FP64 instructions) of the touching and bonded slots,
//                  queued by pair_hamaker. Their two orders are not negatives of each other (the relative
//                  velocity adds the two rotation terms in row order), so both run. One lane per slot, or
//                  three (one spring each) where the queue is short: 20 -> 12 us for 256 monomers.
//   pair_fold      adds each row's slot values in ascending slot order, exactly as the sequential row loop
//                  does, then the half kick and, inside a run of steps, the next step's kick and drift.
// Every slot is written by one thread and every sum has a fixed order, so results do not depend on
// scheduling. Measured (graph-replayed steps with their list builds, us): 32768 monomers, contact + limited Hamaker 445 -> 132
// (kernels 49 / 48 / 16; the kernel before evaluated both orders of every pair, one lane per row, 389);
// 96 sintered aggregates (35,613 monomers) 469 -> 113; 5003 monomers, breaking bonds 189 -> 41; 256
// monomers, all pairs 86 -> 34; 40 monomers, one step per call 37 -> 31 to 34.
#include <algorithm>

#include "lg_compact.cuh"
#include "lg_kernels.h"
#include "lg_pair_fp64.cuh"

namespace lg {

namespace {

constexpr uint32_t kNoRev = 255u;  // the partner's row does not list the slot's row (a truncated row)
constexpr int kPairBlock = 128;    // threads per block of pair_hamaker (fewer for small systems)
constexpr int kTile = 512;         // pairs whose contact candidates a block collects at a time
constexpr int kContactBlock = 64;

// A pair within Hamaker range: its separation x_j - x_i, squared length and slots (e2 < 0: none).
struct HamItem {
    d3 r;
    double d2;
    int64_t e, e2;
};

// The lane's place in a shared list for the warp's lanes with `yes` (one atomic per warp).
__device__ __forceinline__ int warp_place(bool yes, int32_t *count, int lane) {
    const uint32_t bal = __ballot_sync(0xffffffffu, yes);
    int q = 0;
    if (lane == 0 && bal) q = atomicAdd(count, __popc(bal));
    return __shfl_sync(0xffffffffu, q, 0) + __popc(bal & ((1u << lane) - 1u));
}

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

// Classifies the pairs of a block, one per lane, collects those within Hamaker range and evaluates their
// terms with full warps (the others' records are zero). Pairs that are bonded or touch go to the contact queue, both orders: candidates (bonded, within
// reach, or with springs to reset) are collected per block and 32 of them at a time take the reference's
// overlap test, so that the contact kernel's warps hold touching pairs only (aggregates hold monomers at
// contact distance to the last bit, half of which do not touch). VERLET: block b takes the owned slots of its rows; all pairs: pairs [b * per, (b + 1) *
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
    __shared__ int4 cand[kTile];   // contact candidates (i, j, slots of j in i and i in j)
    __shared__ HamItem near[kTile];  // pairs within Hamaker range
    __shared__ int32_t held, nheld;
    if (tid == 0) held = nheld = 0;
    __syncthreads();
    // the contact test of up to 32 candidates: to the queue, or their springs reset
    auto settle = [&](int4 c, bool live) {
        const int64_t i = c.x, j = c.y, e = (int64_t)c.z * n + i;
        const bool both = !VERLET || c.w != (int32_t)kNoRev;
        const int64_t e2 = both ? (int64_t)c.w * n + j : e;
        bool go = false;
        if (live) {
            const uint32_t f1 = PV.flags[e], f2 = PV.flags[e2];
            go = ((f1 | f2) & kBonded) != 0;
            if (!go) {  // contact_force.h:65-69
                const d3 dx = sub(ld4(S.x, i), ld4(S.x, j));
                go = !(2.0 * P.contact.r_part - dot(dx, nrmz(dx)) <= 0);
                if (!go) {  // reset_springs (contact_force.h:69,99-101)
                    const int64_t xs = PV.cap * n;
                    if (f1 & kXiLive) {
#pragma unroll 1
                        for (int q = 0; q < 9; ++q) PV.xi[q * xs + e] = 0.0;
                        PV.flags[e] = f1 & ~kXiLive;
                    }
                    if (both && (f2 & kXiLive)) {
#pragma unroll 1
                        for (int q = 0; q < 9; ++q) PV.xi[q * xs + e2] = 0.0;
                        PV.flags[e2] = f2 & ~kXiLive;
                    }
                }
            }
        }
        // queue places for the warp with one atomic
        const uint32_t b1 = __ballot_sync(0xffffffffu, go), b2 = __ballot_sync(0xffffffffu, go && both);
        if (!b1) return;
        int q = 0;
        if (lane == 0) q = atomicAdd(R.q_n, __popc(b1) + __popc(b2));
        const uint32_t lt = (1u << lane) - 1u;
        q = __shfl_sync(0xffffffffu, q, 0) + __popc(b1 & lt) + __popc(b2 & lt);
        if (go) {
            R.q_i[q] = (int32_t)i;
            R.q_k[q] = c.z;
            if (both) {
                R.q_i[q + 1] = (int32_t)j;
                R.q_k[q + 1] = c.w;
            }
        }
    };
    for (int32_t t0 = 0; t0 < count; t0 += kTile) {
        const int32_t t1 = t0 + kTile < count ? t0 + kTile : count;
        for (int32_t c0 = t0 + tid - lane; c0 < t1; c0 += blockDim.x) {
            const int32_t c = c0 + lane;
            int64_t i = 0, j = 0, e = 0, e2 = -1;
            int32_t k = 0, k2 = 0;
            d3 r = zero3();
            double d2 = 0.0;
            const bool live = c < t1;
            bool touch = false, ham = false;
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
                ham = hm != LG_HAMAKER_NONE && !(hm == LG_HAMAKER_LIMITED && above(d2, P.hamaker_skip_d2));
                if (!ham) {
                    st4(R.rec, e, zero3());
                    if (both) st4(R.rec, e2, zero3());
                }
            }
            if (bm != LG_BINARY_NONE) {
                const int q = warp_place(touch, &held, lane);
                if (touch) cand[q] = make_int4((int32_t)i, (int32_t)j, k, k2);
            }
            if (hm != LG_HAMAKER_NONE) {
                const int q = warp_place(ham, &nheld, lane);
                if (ham) near[q] = HamItem{r, d2, e, e2};
            }
        }
        __syncthreads();
        const int found = held, nfound = nheld;
        for (int q = tid; q < nfound; q += blockDim.x) {
            const HamItem it = near[q];
            const double rn = droot(it.d2);
            d3 a = hamaker_accel_n<FAST>(hm, P.hamaker, P.hc, it.r, rn);
            if (hm == LG_HAMAKER_LIMITED && above(rn, P.hamaker_cut)) a = zero3();
            st4(R.rec, it.e, a);
            if (it.e2 >= 0) st4(R.rec, it.e2, neg(a));
        }
        // (the last warps first: the first ones have the Hamaker list's remainder)
        for (int q = (int)blockDim.x - 32 - (tid - lane); q < found; q += blockDim.x)
            settle(cand[q + lane < found ? q + lane : q], q + lane < found);
        if (t0 + kTile < count) {
            __syncthreads();
            if (tid == 0) held = nheld = 0;
            __syncthreads();
        }
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
        slot_binary_fp64<FAST, CONNECTORS, false>(P, S, PV, BV, n, i, e, j, ld4(S.x, i), ld4(S.v, i), ld4(S.w, i), pb, pbl);
        combine_pair_fp64(true, ham, pb, pbl, ld4(R.rec, e), pa, pal);
        R.rec[e] = make_double4_32a(pa.x, pa.y, pa.z, 1.0);
        st4(R.tq, e, pal);
    }
}

// The same with three lanes per slot, ten slots per warp (see slot_binary_fp64), for queues short enough
// that one slot's chain of FP64 instructions is what a step waits for.
template <bool VERLET, bool FAST>
__global__ void __launch_bounds__(32) pair_contacts_split(Params P, StateView S, PairView PV, BondView BV,
                                                          PairScratch R) {
    const int64_t n = P.n;
    const int32_t total = *R.q_n;
    const bool ham = P.hamaker_model != LG_HAMAKER_NONE;
    const int lane = threadIdx.x, sub = lane % 3;
    if (lane >= 30) return;
    for (int32_t q = blockIdx.x * 10 + lane / 3; q < total; q += gridDim.x * 10) {
        const int64_t i = R.q_i[q], k = R.q_k[q], e = k * n + i;
        const int64_t j = VERLET ? (int64_t)PV.nbr[e] : (k < i ? k : k + 1);
        const int32_t left = total - (q - lane / 3);  // slots of this round's warp
        const uint32_t three = left >= 10 ? 0x3fffffffu : (1u << (3 * left)) - 1u;
        d3 pb, pbl, pa, pal;
        slot_binary_fp64<FAST, false, false, true>(P, S, PV, BV, n, i, e, j, ld4(S.x, i), ld4(S.v, i), ld4(S.w, i), pb,
                                                   pbl, sub, three);
        if (sub == 2) continue;
        combine_pair_fp64(true, ham, pb, pbl, ld4(R.rec, e), pa, pal);
        if (sub == 0) R.rec[e] = make_double4_32a(pa.x, pa.y, pa.z, 1.0);
        else st4(R.tq, e, pal);
    }
}

constexpr int kFoldRows = 10;    // rows per block of pair_fold: three lanes each in two warps
constexpr int kFoldAhead = 16;   // slots whose pair terms a lane of pair_fold has in flight
constexpr int kRowsAhead = 4;    // the same for pair_fold_rows
// pair_fold_rows issues 125 FP64 instructions for 32 rows, pair_fold 30 for ten, in shorter chains, so it wins until
// the rows fill the SMs' sub-partitions, and longer the longer they are. us a step, pair_fold / pair_fold_rows: aggregate
// 12000 rows 53.3 / 59.2, 16384 65.5 / 67.4, 20000 72.5 / 73.7, 26000 84.1 / 82.8; chain 12000 32.4 / 33.1, 16384 39.8 / 38.4,
// 20000 41.7 / 40.0. A body force takes a lane of ten or of 32 rows more: 14000 60.2 / 60.9, 20000 81.1 / 77.3. Facets
// take much more of it: 8000 66.8 / 70.5, 9000 62.6 / 62.3, 10000 80.7 / 70.6, 14000 97.4 / 77.8.
static int64_t fold_rows_from(const Params &P) { return P.n_facets > 0 ? 9000 : 16384; }
// pair_contacts_split issues about 190 FP64 instructions for ten slots instead of 300 for 32, so it wins
// while its warps (0.2 per particle in an aggregate) leave the FP64 units time, less of it the more the contacts slide,
// roll and twist. us a step, split / not, spins of v / r: contacts with Hamaker forces 6100 46.3 / 44.6, 7130 49.5 / 45.4,
// 8300 53.8 / 49.3; bonds without 6100 37.3 / 35.5, 8300 45.3 / 39.1; short queues gain beyond the line (contacts alone,
// which fly apart: 6100 26.7 / 33.4, 8300 27.3 / 34.3). Below it: 256 particles 25.1 / 31.8, 5000 34.3 / 39.2, no spins.
constexpr int64_t kSplitUpTo = 6000;

// Small systems: lane 3 r + c of the first warp sums force component c of the block's row r in slot order,
// one dependent chain per lane with the loads of slots kFoldAhead ahead issued between its additions (a
// dependent FP64 addition takes about 34 ns); the second warp does the same for the torques, which only
// records with a binary part carry (tag 1). (A zero added to a sum that started at +0 leaves its bits.)
template <bool VERLET, bool FACETS>
__global__ void __launch_bounds__(64) pair_fold(Params P, StateView S, PairView PV, BondView BV, PairScratch R,
                                                double hdt, double dt, int move_facets, int kick) {
    __shared__ double row[kFoldRows][12];
    const int64_t n = P.n;
    if (move_facets && blockIdx.x == 0 && threadIdx.x == 0) compact::move_facets(P, S, dt);
    if (blockIdx.x == 0 && threadIdx.x == 31) *R.q_n = 0;  // the next evaluation's queue
    const int lane = threadIdx.x & 31;
    const bool torque = threadIdx.x >= 32;
    const int r = lane / 3, c = lane % 3;
    const int64_t i = (int64_t)blockIdx.x * kFoldRows + r;
    const bool mine = r < kFoldRows && i < n;
    double sum = 0.0, vel = 0.0;
    uint32_t h = 0;
    if (mine) {
        const int64_t len = VERLET ? (int64_t)PV.row_len[i] : n - 1;
        vel = reinterpret_cast<const double *>(torque ? S.w : S.v)[4 * i + c];
        h = hold_of(P.hold, i);
        const int64_t pitch = 4 * n;
        const double *col = reinterpret_cast<const double *>(R.rec) + 4 * i + (torque ? 3 : c);
        double t[kFoldAhead];
#pragma unroll
        for (int q = 0; q < kFoldAhead; ++q) t[q] = q < len ? col[q * pitch] : 0.0;
        if (!torque) {
            for (int64_t k = 0; k < len; k += kFoldAhead) {
#pragma unroll
                for (int q = 0; q < kFoldAhead; ++q) {
                    const int64_t kk = k + kFoldAhead + q;
                    sum += t[q];
                    t[q] = kk < len ? col[kk * pitch] : 0.0;
                }
            }
        } else {
            const double *tq = reinterpret_cast<const double *>(R.tq) + 4 * i + c;
            for (int64_t k = 0; k < len; k += kFoldAhead) {
                uint32_t tags = 0;
#pragma unroll
                for (int q = 0; q < kFoldAhead; ++q) {
                    const int64_t kk = k + kFoldAhead + q;
                    if (__double_as_longlong(t[q]) != 0) tags |= 1u << q;
                    t[q] = kk < len ? col[kk * pitch] : 0.0;
                }
                for (; tags; tags &= tags - 1) sum += tq[(k + __ffs(tags) - 1) * pitch];
            }
        }
    }
    const int c6 = torque ? 3 + c : c;
    if (FACETS) {  // unary terms of the whole row, on the row's first lane
        if (mine) {
            row[r][c6] = sum;
            row[r][6 + c6] = vel;
        }
        __syncthreads();
        if (mine && c6 == 0) {
            double *w = row[r];
            d3 ua, ual;
            if (compact::unary_terms(P, S, i, n, mk3(w[6], w[7], w[8]), mk3(w[9], w[10], w[11]), ua, ual)) {
                w[0] += ua.x;
                w[1] += ua.y;
                w[2] += ua.z;
                w[3] += ual.x;
                w[4] += ual.y;
                w[5] += ual.z;
            }
        }
        __syncthreads();
        if (mine) sum = row[r][c6];
    }
    const bool hv = h & (torque ? LG_HOLD_OMEGA : LG_HOLD_V);
    double v1 = vel;
    if (mine) {
        reinterpret_cast<double *>(torque ? S.al : S.a)[4 * i + c] = sum;
        if (!isfinite(sum)) set_error(S.err, LG_DEVERR_NONFINITE);
        if (!hv) v1 = vel + hdt * sum;
        if (kick && !hv) v1 = v1 + hdt * sum;  // the next step's opening half kick
        reinterpret_cast<double *>(torque ? S.w_out : S.v_out)[4 * i + c] = v1;
    }
    if (!kick) return;
    if (!BV.cn) {  // the next step's drift of this component
        if (mine && !(h & (torque ? LG_HOLD_THETA : LG_HOLD_X))) {
            double *p = reinterpret_cast<double *>(torque ? S.th : S.x) + 4 * i + c;
            *p = *p + dt * v1;
        }
        return;
    }
    // with connectors the drift needs the whole particle
    __syncthreads();
    if (mine) row[r][c6] = v1;
    __syncthreads();
    if (mine && c6 == 0)
        drift_one(n, i, S.x, S.th, mk3(row[r][0], row[r][1], row[r][2]), mk3(row[r][3], row[r][4], row[r][5]), dt, BV, h);
}

// Large systems: one lane per row, all its components (three additions a slot for 32 rows instead of one
// for five, so the fewest FP64 instructions; there are enough rows to fill the SMs). The tagged slots'
// torques are added after each 32 slots' forces.
template <bool VERLET, bool FACETS>
__global__ void __launch_bounds__(32) pair_fold_rows(Params P, StateView S, PairView PV, BondView BV,
                                                             PairScratch R, double hdt, double dt, int move_facets,
                                                             int kick) {
    const int64_t n = P.n;
    if (move_facets && blockIdx.x == 0 && threadIdx.x == 0) compact::move_facets(P, S, dt);
    if (blockIdx.x == 0 && threadIdx.x == 0) *R.q_n = 0;  // the next evaluation's queue
    const int64_t i = blockIdx.x * (int64_t)32 + threadIdx.x;
    if (i >= n) return;
    const int64_t len = VERLET ? (int64_t)PV.row_len[i] : n - 1;
    const d3 vi = ld4(S.v, i), wi = ld4(S.w, i);
    const dbl4 *rec = R.rec + i, *tq = R.tq + i;
    const dbl4 zero = make_double4_32a(0.0, 0.0, 0.0, 0.0);
    d3 acc = zero3(), accw = zero3();
    dbl4 t[kRowsAhead], u[kRowsAhead];
#pragma unroll
    for (int q = 0; q < kRowsAhead; ++q) t[q] = q < len ? rec[q * n] : zero;
    for (int64_t k0 = 0; k0 < len; k0 += 32) {
        uint32_t tags = 0;
        for (int k = 0; k < 32 && k0 + k < len; k += kRowsAhead) {
#pragma unroll
            for (int q = 0; q < kRowsAhead; ++q) {
                const int64_t kk = k0 + k + kRowsAhead + q;
                u[q] = kk < len ? rec[kk * n] : zero;
            }
#pragma unroll
            for (int q = 0; q < kRowsAhead; ++q) {
                acc = add(acc, mk3(t[q].x, t[q].y, t[q].z));
                if (__double_as_longlong(t[q].w) != 0) tags |= 1u << (k + q);
                t[q] = u[q];
            }
        }
        for (; tags; tags &= tags - 1) accw = add(accw, ld4(tq, (k0 + __ffs(tags) - 1) * n));
    }
    compact::finish_row<FACETS>(P, S, i, n, acc, accw, vi, wi, hdt);
    if (kick) {  // the next step's opening half kick and drift, as kick_drift_fp64
        const uint32_t h = hold_of(P.hold, i);
        const d3 v2 = kick_unless(kick_unless(vi, hdt, acc, h & LG_HOLD_V), hdt, acc, h & LG_HOLD_V);
        const d3 w2 = kick_unless(kick_unless(wi, hdt, accw, h & LG_HOLD_OMEGA), hdt, accw, h & LG_HOLD_OMEGA);
        st4(S.v_out, i, v2);
        st4(S.w_out, i, w2);
        drift_one(n, i, S.x, S.th, v2, w2, dt, BV, h);
    }
}

// Rows per block of owned slots: blocks enough for every SM, yet full batches of 32, and at most the 32 rows whose
// partners fill a tile. us a step, 4 / 8 / 16 / 32 rows: aggregates of 2000 28.4 / 31.4 / 29.5 / 39.2, 3000 29.4 / 32.2 /
// 30.7 / 39.5, 4000 32.1 / 33.2 / 31.6 / 40.0, 8000 49.6 / 46.7 / 43.1 / 50.3; 16 / 32 rows: 12000 45.9 / 53.3, 16384 63.3 /
// 65.5, 20000 71.9 / 72.5, 30000 96.3 / 93.5, without Hamaker forces 12000 33.3 / 33.7, 16384 43.3 / 41.0, 30000 55.8 / 52.5;
// 4 / 16 rows: chain of 2600 23.9 / 23.2, of 3300 24.6 / 23.5.
int32_t pair_block_rows(int64_t n) { return n >= 16384 ? 32 : n >= 2500 ? 16 : 4; }

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
            if (R.rb == 4) threads = 64;
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
        } else if (n <= kSplitUpTo) {
            const unsigned warps = (unsigned)std::min<int64_t>((std::min<int64_t>(slots, 4 * n) + 9) / 10, 152 * 16);
            if (verlet) pair_contacts_split<true, FAST><<<warps, 32, 0, st>>>(P, S, PV, BV, R);
            else pair_contacts_split<false, FAST><<<warps, 32, 0, st>>>(P, S, PV, BV, R);
        } else {
            if (verlet) pair_contacts<true, FAST, false><<<blocks, kContactBlock, 0, st>>>(P, S, PV, BV, R);
            else pair_contacts<false, FAST, false><<<blocks, kContactBlock, 0, st>>>(P, S, PV, BV, R);
        }
        ++kernels;
    }
    const bool unary = P.n_facets > 0 || P.ext_a, rows = n >= fold_rows_from(P);
    const int64_t per = rows ? 32 : kFoldRows;
    const unsigned fb = (unsigned)((n + per - 1) / per);
    auto fold = rows ? (verlet ? (unary ? pair_fold_rows<true, true> : pair_fold_rows<true, false>)
                               : (unary ? pair_fold_rows<false, true> : pair_fold_rows<false, false>))
                     : (verlet ? (unary ? pair_fold<true, true> : pair_fold<true, false>)
                               : (unary ? pair_fold<false, true> : pair_fold<false, false>));
    fold<<<fb, rows ? 32 : 64, 0, st>>>(P, S, PV, BV, R, hdt, dt, move_facets, kick ? 1 : 0);
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
