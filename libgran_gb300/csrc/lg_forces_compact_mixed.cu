// lg_forces_compact_mixed.cu -- force evaluation of the mixed-precision path (sm_103a): contacts,
// Hamaker pairs and unary terms on three streams, then a completion; slot layout and flags shared
// with the FP64 path.
//
//   mixed_contacts         contact and bond pairs of listed systems, each unordered pair once: the owned
//                          contact candidates (near_owners, after each list build) are queued per block and
//                          evaluated a warp at a time; each order's accelerations go to a record per
//                          candidate, which the completion adds per row in entry order.
//   forces_contacts_mixed  contact and bond pairs row by row: the lists whose candidates are too many for that
//                          (near_scratch in lg_engine.cpp), all pairs, and systems whose two orders of a pair
//                          may break differently. Candidates are queued per warp (ballot
//                          order) and evaluated 32 at a time, folded per row in slot order into
//                          float-float sums (MixedExtra::csum).
//   forces_hamaker_mixed   Hamaker pairs over all slots, in windows of four slots held in registers, L
//                          lanes per row; the windows' sums are added in the order that the slicing
//                          defines. Runs beside the contact kernel (two streams).
//   forces_hamaker_all     the same over all pairs of large systems, a lane per row.
//   unary_mixed            facet and body terms (FP64), on a third stream.
//   forces_finish_ff       completion inside a run of steps (no facets, no body term): the sums, the
//                          end-of-step half kick, the next step's half kick and drift, all in
//                          float-float on the FP32 pipes; the run's last step writes the FP64 state.
//   forces_finish_mixed    the FP64 completion (facets, body terms, single steps): contact part +
//                          Hamaker part to FP64, the unary terms added, stores, half kick (+ next kick
//                          and drift).
//
// The per-pair and per-row pieces (and the precision scheme) are in lg_mixed_pairs.cuh, shared with
// the persistent step kernel (lg_step_mixed.cu). Per-row sums are in an order fixed by the row
// alone, so a system gives the same bits alone and inside a batch (with the same slicing).
#include <algorithm>
#include <cstddef>

#include "lg_launch.cuh"
#include "lg_mixed_pairs.cuh"

namespace lg {

using namespace mixed;

namespace {

constexpr uint32_t kNoPartner = 255u;  // the partner's row does not list the entry's row

// ---- launch shapes of the two-stream kernels ----
// Slices per row group of the Hamaker kernel: 0 chooses from the launch size (compile-time
// override for tuning).
#ifndef LG_MIXED_SLICES
#define LG_MIXED_SLICES 0
#endif
constexpr int kCWarps = 2;   // warps per block
constexpr int kHThreads = 128;  // threads per block of the Hamaker kernel
// Resident blocks per SM that forces_contacts_mixed is compiled for: 8 leave it the 128 registers that it needs.
// With 12 (80 registers, for more warps of the Hamaker kernel beside it) it spilled, and was slower at every size
// and list length measured beside that kernel (us a step, 8 / 12 blocks, list radius 4.5 r and 6 r: 1000 monomers
// 13.7 / 16.2 and 16.6 / 20.9, 32768 26.3 / 30.0 and 38.2 / 46.0) as well as alone.
constexpr int kCBlocks = 8;
}  // namespace

// Contact and bond pairs of rows row0 .. row0 + 32/T - 1 per warp (contact_rows), csum receives the
// contact part of the row's accelerations.
template <bool NEAR, int T>
__global__ void __launch_bounds__(kCWarps * 32, kCBlocks)
    forces_contacts_mixed(Params P, StateView S, PairView PV, BondView BV, MixedExtra MX) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kRows = 32 / T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ContactSmem &W = reinterpret_cast<ContactSmem *>(smem_raw)[warp];
    contact_rows<NEAR, T>(P, PV, BV, MX, W, ((int64_t)blockIdx.x * kCWarps + warp) * kRows, lane);
}

// The owned contact candidates of each block of `rb` rows: of the two entries of a pair (i, j) the one in
// row i when i < j and i + j is odd, or i > j and i + j is even; an entry that the partner's row does not
// list is always owned. (j; local row, slot, slot in the partner's row; entry, entry in the partner's row.)
__global__ void __launch_bounds__(512) near_owners(int64_t n, PairView PV, NearScratch R) {
    __shared__ int32_t cnt;
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    const int64_t row0 = (int64_t)blockIdx.x * R.rb;
    uint4 *own = R.own + row0 * PV.cap;
    const int per = blockDim.x / R.rb;  // lanes per row
    const int r = threadIdx.x % R.rb;
    const int64_t i = row0 + r;
    const int len = i < n ? PV.near_len[i] : 0;
    for (int m = threadIdx.x / R.rb; m < len; m += per) {
        const int32_t j = PV.near_j[(int64_t)m * n + i];
        const uint32_t k = PV.near_k[(int64_t)m * n + i];
        const int lj = PV.near_len[j];
        int m2 = 0;
        while (m2 < lj && PV.near_j[(int64_t)m2 * n + j] != (int32_t)i) ++m2;
        const bool both = m2 < lj;
        if (both && !(((i + j) & 1) ? i < j : i > j)) continue;
        const uint32_t k2 = both ? PV.near_k[(int64_t)m2 * n + j] : kNoPartner;
        own[atomicAdd(&cnt, 1)] =
            make_uint4((uint32_t)j, (uint32_t)r | (k << 8) | (k2 << 16), (uint32_t)m | ((uint32_t)m2 << 8), 0u);
    }
    __syncthreads();
    if (threadIdx.x == 0) R.own_n[blockIdx.x] = cnt;
}

// Contact and bond pairs, each evaluated once for both of its rows (contact_pair): the block's owned
// candidates are classified two per thread, those that can touch or are bonded are queued in shared memory and
// evaluated 32 at a time. Each entry's accelerations go to its record (zero when apart), which the
// completion adds per row in entry order; the springs of both slots are written.
// What bounds it: instruction issue and the latency of its gathers.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    mixed_contacts(Params P, PairView PV, BondView BV, MixedExtra MX, NearScratch R) {
    struct Item {
        int32_t i, j;
        uint32_t kk, mm;  // slots (k | k2 << 8), entries (m | m2 << 8); k2 = kNoPartner: one-sided
    };
    __shared__ Item queue[4 * THREADS];
    __shared__ int32_t qn;
    const int tid = threadIdx.x;
    const int64_t n = P.n;
    const int count = R.own_n[blockIdx.x];
    const int64_t row0 = (int64_t)blockIdx.x * R.rb;
    const uint4 *own = R.own + row0 * PV.cap;
    const int64_t xs = PV.cap * n, bs = (int64_t)BV.bcap * n;
    auto put = [&](int64_t i, uint32_t m, float4 a, float4 b) {
        R.rec[2 * ((int64_t)m * n + i)] = a;
        R.rec[2 * ((int64_t)m * n + i) + 1] = b;
    };
    auto part = [&](int64_t i, uint32_t m, int64_t e, uint32_t fl) {  // reset_springs (contact_force.h:69,99-101)
        put(i, m, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f));
        if (!(fl & kXiLive)) return;
#pragma unroll
        for (int c = 0; c < 9; ++c) PV.xi[spring_at(PV.aos, c, e, xs)] = 0.0;
        PV.flags[e] = fl & ~kXiLive;
    };
    for (int t0 = 0; t0 < count; t0 += 2 * THREADS) {
        if (tid == 0) qn = 0;
        __syncthreads();
        uint4 o[2];
        bool live[2];
        float4 pi[2], pj[2];
        uint32_t fl[2], fl2[2];
        int64_t e[2], e2[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            live[u] = t0 + u * THREADS + tid < count;
            o[u] = own[live[u] ? t0 + u * THREADS + tid : 0];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t j = o[u].x, i = row0 + (o[u].y & 0xffu);
            const uint32_t k = (o[u].y >> 8) & 0xffu, k2 = (o[u].y >> 16) & 0xffu;
            e[u] = (int64_t)k * n + i;
            e2[u] = k2 != kNoPartner ? (int64_t)k2 * n + j : e[u];
            pi[u] = MX.x32[2 * i];
            pj[u] = MX.x32[2 * j];
            fl[u] = PV.flags[e[u]];
            fl2[u] = PV.flags[e2[u]];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (!live[u]) continue;
            const int64_t j = o[u].x, i = row0 + (o[u].y & 0xffu);
            const uint32_t k = (o[u].y >> 8) & 0xffu, k2 = (o[u].y >> 16) & 0xffu, m = o[u].z & 0xffu, m2 = o[u].z >> 8;
            const bool both = k2 != kNoPartner;
            const float dx = pi[u].x - pj[u].x, dy = pi[u].y - pj[u].y, dz = pi[u].z - pj[u].z;
            if (((fl[u] | fl2[u]) & kBonded) || fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= MX.contact2f) {
                // the two orders' states agree, unless only one of them lost its bond or list place
                const bool split = both && ((fl[u] ^ fl2[u]) & (kBonded | kXiLive));
                const int q = atomicAdd(&qn, split ? 2 : 1);
                queue[q] = Item{(int32_t)i, (int32_t)j, k | ((split ? kNoPartner : k2) << 8), m | (m2 << 8)};
                if (split) queue[q + 1] = Item{(int32_t)j, (int32_t)i, k2 | (kNoPartner << 8), m2 | (m << 8)};
            } else {
                part(i, m, e[u], fl[u]);
                if (both) part(j, m2, e2[u], fl2[u]);
            }
        }
        __syncthreads();
        const int total = qn;
        for (int q = tid; q < total; q += THREADS) {
            const Item it = queue[q];
            const int64_t i = it.i, j = it.j;
            const uint32_t k = it.kk & 0xffu, k2 = it.kk >> 8;
            const bool both = k2 != kNoPartner;
            const int64_t e = (int64_t)k * n + i, e2 = both ? (int64_t)k2 * n + j : e;
            const uint32_t fl = PV.flags[e], fl2 = PV.flags[e2];
            const bool bonded = (fl & kBonded) != 0;
            // (mixed precision stores springs as one 9-component record per slot or bond)
            const int64_t at = bonded ? (int64_t)bond_slot_of(fl) * n + i : e;
            const int64_t at2 = bonded ? (int64_t)bond_slot_of(fl2) * n + j : e2;
            float2 *store = reinterpret_cast<float2 *>(bonded ? BV.xi : PV.xi);
            const int32_t aos = bonded ? BV.aos : PV.aos;
            const int64_t stride = bonded ? bs : xs;
            const Body bi = body_of(MX, n, i), bj = body_of(MX, n, j);
            ff s[3][3] = {};  // springs of a slot that is not live are zero
            if (fl & (kBonded | kXiLive))
#pragma unroll
                for (int c = 0; c < 9; ++c) {
                    const float2 v = store[spring_at(aos, c, at, stride)];
                    s[c / 3][c % 3] = ff{v.x, v.y};
                }
            ContactOut o;
            if (!contact_pair(P, MX, bonded, i, j, bi, bj, s, o)) {
                part(i, it.mm & 0xffu, e, fl);
                if (both) part(j, it.mm >> 8, e2, fl2);
                continue;
            }
            const bool breaks = bonded && P.binary_model == LG_BINARY_BREAKING_SINTER;
            const float f2 = fdot(o.force, o.force);
            float sgn = 1.0f;
            const int sides = both ? 2 : 1;
#pragma unroll 1
            for (int side = 0; side < sides; ++side) {  // the row's own values, then the partner's
                const int64_t row = side ? j : i, es = side ? e2 : e, as = side ? at2 : at;
                const uint32_t f = side ? fl2 : fl, m = side ? it.mm >> 8 : it.mm & 0xffu;
#pragma unroll
                for (int c = 0; c < 9; ++c) {
                    const ff v = s[c / 3][c % 3];
                    const float g = c / 3 == 1 ? 1.0f : sgn;
                    store[spring_at(aos, c, as, stride)] = make_float2(g * v.hi, g * v.lo);
                }
                const f3 fo = fm(sgn * o.force.x, sgn * o.force.y, sgn * o.force.z);
                const f3 roll = fm(sgn * o.roll.x, sgn * o.roll.y, sgn * o.roll.z);
                const f3 twist = fm(sgn * o.twist.x, sgn * o.twist.y, sgn * o.twist.z);
                const f3 tau = torque_of(roll, o.slide, twist, o.rr, o.rp);
                put(row, m, make_float4(fo.x * MX.bin_im, fo.y * MX.bin_im, fo.z * MX.bin_im, tau.x * MX.bin_iI),
                    make_float4(tau.y * MX.bin_iI, tau.z * MX.bin_iI, 0.f, 0.f));
                if (breaks) {
                    const float st = (float)BV.strength[as];
                    if (f2 > st * st) {
                        BV.intact[as] = 0;
                        PV.flags[es] = f & ~(kBonded | (0xffu << 8));
                    }
                } else if (!(f & (kBonded | kXiLive))) {
                    PV.flags[es] = f | kXiLive;
                }
                sgn = -1.0f;
            }
        }
        __syncthreads();
    }
}

// Contact part of row i's accelerations from its entries' records: T running sums over entries 0, T, ...
// and 1, T + 1, ..., then added in order (the order in which contact_rows with T lanes per row adds them).
template <int T>
__device__ __forceinline__ void contact_sums(const PairView &PV, const NearScratch &R, int64_t n, int64_t i,
                                             ff (&a)[3], ff (&al)[3]) {
    ff acc[T][6];
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[t][c] = ff{0.f, 0.f};
    constexpr int kAhead = 4;  // entries loaded with the row's count, before it is known (every row has them)
    float4 p[kAhead], q[kAhead];
    const int len = PV.near_len[i];
    const bool ahead = PV.cap >= kAhead;
    for (int m = 0; m == 0 || m < len; m += kAhead) {
#pragma unroll
        for (int t = 0; t < kAhead; ++t) {
            if (m == 0 ? ahead || t < len : m + t < len) {
                const float4 *rec = R.rec + 2 * ((int64_t)(m + t) * n + i);
                p[t] = rec[0];
                q[t] = rec[1];
            }
        }
#pragma unroll
        for (int t = 0; t < kAhead; ++t) {
            if (m + t < len) {
                ff(&s)[6] = acc[t % T];
                ff_acc(s[0], p[t].x);
                ff_acc(s[1], p[t].y);
                ff_acc(s[2], p[t].z);
                ff_acc(s[3], p[t].w);
                ff_acc(s[4], q[t].x);
                ff_acc(s[5], q[t].y);
            }
        }
    }
#pragma unroll
    for (int t = 1; t < T; ++t)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            ff_acc(acc[0][c], acc[t][c].hi);
            ff_acc(acc[0][c], acc[t][c].lo);
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        a[c] = acc[0][c];
        al[c] = acc[0][3 + c];
    }
}

// The contact part of row i: from the records (R.rec) or from the contact kernel's sums (MX.csum).
__device__ __forceinline__ void contact_part(const PairView &PV, const NearScratch &R, const MixedExtra &MX, int64_t n,
                                             int64_t i, ff (&a)[3], ff (&al)[3]) {
    if (R.rec) {
        if (R.lanes == 2) contact_sums<2>(PV, R, n, i, a, al);
        else contact_sums<1>(PV, R, n, i, a, al);
        return;
    }
    const float4 c0 = MX.csum[3 * i], c1 = MX.csum[3 * i + 1], c2 = MX.csum[3 * i + 2];
    a[0] = ff{c0.x, c0.y};
    a[1] = ff{c0.z, c0.w};
    a[2] = ff{c1.x, c1.y};
    al[0] = ff{c1.z, c1.w};
    al[1] = ff{c2.x, c2.y};
    al[2] = ff{c2.z, c2.w};
}

// Hamaker pairs: hsum receives the Hamaker part of the row's acceleration as a float-float sum. L lanes
// per row, lane l taking windows l, l + L, ... of kWin slots and evaluating their pairs from registers
// (the partner indices of its next window are loaded meanwhile). The windows' sums are added in the order
// that SL slices define, whatever L is: slice s adds windows s, s + SL, ... one after another, then the
// slices are added in order.
template <bool VERLET, int HM, int L, int SL>
__global__ void __launch_bounds__(kHThreads, L == 1 ? 6 : 7) forces_hamaker_mixed(Params P, PairView PV, MixedExtra MX) {
    static_assert(L % SL == 0 && 32 % L == 0, "a row's lanes hold whole slices");
    const int lane = threadIdx.x & 31, l = lane % L, base = lane - l;
    const int64_t n = P.n;
    const int64_t i = ((int64_t)blockIdx.x * kHThreads + threadIdx.x) / L;
    const bool active = i < n;
    int32_t len = 0;
    float4 xh = make_float4(0.f, 0.f, 0.f, 0.f), xl = xh;
    if (active) {
        len = VERLET ? PV.row_len[i] : (int32_t)(n - 1);
        xh = MX.x32[2 * i];
        xl = MX.x32[2 * i + 1];
    }
    const int32_t maxlen = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)len);
    ff acc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};  // of slice l % SL
    int32_t jn[kWin];
    window_partners<VERLET>(PV, n, i, len, l * kWin, jn);
    for (int32_t k0 = 0; k0 < maxlen; k0 += L * kWin) {
        int32_t j[kWin];
#pragma unroll
        for (int u = 0; u < kWin; ++u) j[u] = jn[u];
        window_partners<VERLET>(PV, n, i, len, k0 + (L + l) * kWin, jn);
        const f3 w = window_sum<HM>(MX, xh, xl, j);
        if (L == SL) {
            ff_acc(acc[0], w.x);
            ff_acc(acc[1], w.y);
            ff_acc(acc[2], w.z);
        } else {
#pragma unroll
            for (int t = 0; t < L / SL; ++t) {
                const int src = base + l % SL + t * SL;
                ff_acc(acc[0], __shfl_sync(0xffffffffu, w.x, src));
                ff_acc(acc[1], __shfl_sync(0xffffffffu, w.y, src));
                ff_acc(acc[2], __shfl_sync(0xffffffffu, w.z, src));
            }
        }
    }
#pragma unroll
    for (int q = 1; q < SL; ++q) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float hi = __shfl_sync(0xffffffffu, acc[c].hi, base + q), lo = __shfl_sync(0xffffffffu, acc[c].lo, base + q);
            if (l == 0) {
                ff_acc(acc[c], hi);
                ff_acc(acc[c], lo);
            }
        }
    }
    if (!active || l != 0) return;
    MX.hsum[2 * i] = make_float4(acc[0].hi, acc[0].lo, acc[1].hi, acc[1].lo);
    MX.hsum[2 * i + 1] = make_float4(acc[2].hi, acc[2].lo, 0.f, 0.f);
}

// All pairs of large systems: a lane per row and a warp per slice, so that the lanes of a warp read the same
// partners (one broadcast a load; with lanes along a row every lane reads a sector of its own, and those loads
// are what takes the time). The sums are added in the same order.
template <int HM, int SL>
__global__ void __launch_bounds__(32 * SL, 2) forces_hamaker_all(Params P, PairView PV, MixedExtra MX) {
    __shared__ float part[SL][6][32];
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int64_t row0 = (int64_t)blockIdx.x * 32, i = row0 + lane;
    ff acc[3];
    hamaker_rows<false, HM, HM == LG_HAMAKER_LIMITED>(P, PV, MX, row0, sl, SL, lane, acc);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        part[sl][2 * c][lane] = acc[c].hi;
        part[sl][2 * c + 1][lane] = acc[c].lo;
    }
    __syncthreads();
    if (sl != 0 || i >= P.n) return;
    for (int q = 1; q < SL; ++q)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            ff_acc(acc[c], part[q][2 * c][lane]);
            ff_acc(acc[c], part[q][2 * c + 1][lane]);
        }
    MX.hsum[2 * i] = make_float4(acc[0].hi, acc[0].lo, acc[1].hi, acc[1].lo);
    MX.hsum[2 * i + 1] = make_float4(acc[2].hi, acc[2].lo, 0.f, 0.f);
}

// Unary terms (facets, body force) of every particle, beside the pair kernels: they need the FP64 state only,
// and the FP64 pipe, which the pair kernels leave idle (in the completion they took 105 of its 119 us for
// 141,000 particles on a wall). The grid holds no more than sixteen warps per SM, at 64 registers: the FP64
// pipe is nearly as busy as with more, and the rest of the register file is the pair kernels' (restructuring
// batch of 141,000 particles, us a step: 175 with one block per 64 particles at 150 registers, 170 with six
// such blocks per SM, 146 at 80 registers). The facets' edges are formed once per block.
constexpr int kUnaryThreads = 64;
constexpr int kUnaryBlocks = 152 * 8;
__global__ void __launch_bounds__(kUnaryThreads, 16) unary_mixed(Params P, StateView S, MixedExtra MX) {
    __shared__ FacetEdges edges[kMaxFacets];
    if ((int)threadIdx.x < 3 * P.n_facets)
        facet_edge(S.facet_vert + 9 * (threadIdx.x / 3), threadIdx.x % 3, edges[threadIdx.x / 3]);
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)kUnaryThreads + threadIdx.x; i < P.n; i += (int64_t)gridDim.x * kUnaryThreads) {
        if (inactive_of(P.hold, i)) continue;
        d3 ua = zero3(), ual = zero3();
        compact::unary_terms(P, S, i, P.n, ld4(S.v, i), ld4(S.w, i), ua, ual, edges);
        st4(MX.un_a, i, ua);
        st4(MX.un_al, i, ual);
    }
}

// Completion of row i in FP64: contact part (csum when `contacts`) plus the Hamaker part (hsum when
// `hamaker`), both converted to FP64, then the unary terms, stores and half kick; with `kick` also
// the next step's opening half kick and drift, and the float-float copies of the new state.
template <bool FACETS>
__device__ __forceinline__ void finish_fp64_row(const Params &P, const StateView &S, int64_t i, double hdt, double dt,
                                                int contacts, int hamaker, int kick, const MixedExtra &MX,
                                                const PairView &PV, const NearScratch &R) {
    // every input is loaded before anything is stored (the buffers are distinct)
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    ff ac[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}}, alc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    if (contacts) contact_part(PV, R, MX, P.n, i, ac, alc);
    const float4 h0 = hamaker ? MX.hsum[2 * i] : z4, h1 = hamaker ? MX.hsum[2 * i + 1] : z4;
    const d3 vi = ld4(S.v, i), wi = ld4(S.w, i);
    d3 xo = zero3(), tho = zero3();
    if (kick) {
        xo = ld4(S.x, i);
        tho = ld4(S.th, i);
    }
    // contact part (float-float pairs hi, lo), then the Hamaker part
    d3 a_tot = mk3(ff_to_d(ac[0]), ff_to_d(ac[1]), ff_to_d(ac[2]));
    d3 al_tot = mk3(ff_to_d(alc[0]), ff_to_d(alc[1]), ff_to_d(alc[2]));
    if (hamaker) {
        const d3 ah = mk3((double)h0.x + (double)h0.y, (double)h0.z + (double)h0.w, (double)h1.x + (double)h1.y);
        a_tot = contacts ? add(a_tot, ah) : ah;
    }
    if (FACETS) {  // (unary_mixed's terms)
        a_tot = add(a_tot, ld4(MX.un_a, i));
        al_tot = add(al_tot, ld4(MX.un_al, i));
    }
    compact::finish_row<false>(P, S, i, P.n, a_tot, al_tot, vi, wi, hdt);
    if (kick) {  // the next step's opening half kick and drift (the end-of-step velocities are not kept)
        const uint32_t h = hold_of(P.hold, i);
        const bool hv = h & LG_HOLD_V, hw = h & LG_HOLD_OMEGA;
        const d3 vh = kick_unless(kick_unless(vi, hdt, a_tot, hv), hdt, a_tot, hv);
        const d3 wh = kick_unless(kick_unless(wi, hdt, al_tot, hw), hdt, al_tot, hw);
        st4(S.v_out, i, vh);
        st4(S.w_out, i, wh);
        const d3 xn = (h & LG_HOLD_X) ? xo : add(xo, scl(dt, vh));
        const d3 thn = (h & LG_HOLD_THETA) ? tho : add(tho, scl(dt, wh));
        if (!(h & LG_HOLD_X)) st4(S.x, i, xn);
        if (!(h & LG_HOLD_THETA)) st4(S.th, i, thn);
        rel_ff(xn, MX.ox, MX.oy, MX.oz, MX.agg, MX.orig, i, P.n, MX.x32);
        state_ff(vh, wh, i, P.n, MX.v32, MX.s32);
    }
}

template <bool FACETS>
__global__ void __launch_bounds__(64) forces_finish_mixed(Params P, StateView S, double hdt, double dt,
                                                          int move_facets, int contacts, int hamaker, int kick,
                                                          MixedExtra MX, PairView PV, NearScratch R) {
    if (move_facets && blockIdx.x == 0 && threadIdx.x == 0) compact::move_facets(P, S, dt);
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= P.n || inactive_of(P.hold, i)) return;
    finish_fp64_row<FACETS>(P, S, i, hdt, dt, contacts, hamaker, kick, MX, PV, R);
}

// Completion of a step of a run (no facets, no body term), integrating in float-float on the FP32
// pipes: between the first and the last step of a run the state lives in x32 / v32 / s32 (the FP64
// x and theta keep the values of the run's first step, v and omega are left behind) and the last
// step writes the FP64 state. Velocities and spins are float-float values (about 2^-46 of their
// magnitude). Positions are carried twice: x32 (relative to the system origin) advances for the
// force kernels, and the displacement since the run's first step accumulates from zero in s32, so
// that the last step's FP64 position x_first + displacement is not limited by the float-float
// resolution of x32 (a step moves a particle by about 1e-9 of its distance from the origin); the
// rotation theta accumulates the same way.
//   LAST = false: the end-of-step half kick, the next step's opening half kick and drift;
//   LAST = true:  the end-of-step half kick, then a, alpha, v, omega, x and theta in FP64.
// s32: [i] low parts of omega; [n + i] / [2n + i] displacement hi / lo; [3n + i] / [4n + i]
// rotation hi / lo.
template <bool LAST>
__global__ void __launch_bounds__(64) forces_finish_ff(Params P, StateView S, int contacts, int hamaker, ff hdt, ff dt,
                                                       double hdt_d, double dt_d, MixedExtra MX, PairView PV,
                                                       NearScratch R) {
    const int64_t n = P.n;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t h = hold_of(P.hold, i);
    if (h & kHoldInactive) return;  // takes no part
    if (h) {  // a held particle keeps its FP64 state current (a held value stays exactly as it was)
        finish_fp64_row<false>(P, S, i, hdt_d, dt_d, contacts, hamaker, LAST ? 0 : 1, MX, PV, R);
        return;
    }
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 h0 = hamaker ? MX.hsum[2 * i] : z4, h1 = hamaker ? MX.hsum[2 * i + 1] : z4;
    ff a[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}}, al[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    if (contacts) contact_part(PV, R, MX, n, i, a, al);
    if (hamaker) {
        const ff ah[3] = {{h0.x, h0.y}, {h0.z, h0.w}, {h1.x, h1.y}};
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] = contacts ? ff_add(a[c], ah[c]) : ah[c];
    }
    finish_ff_plain<LAST>(S, i, n, a, al, hdt, dt, MX, MX.x32, MX.v32);
}

namespace {

// Lanes per row of the contact kernel: T = 2 (or 1, a tuning choice that suits large batches) for
// candidate lists (a few entries per row); a whole warp per row for all pairs (n - 1 candidates per
// row: the lanes share them, and the row count no longer bounds the warps a small system can use).
template <bool NEAR, int T>
void launch_contacts(const Params &P, const StateView &S, const PairView &PV, const BondView &BV, const MixedExtra &MX,
                     cudaStream_t st, int share) {
    const size_t smem = sizeof(ContactSmem) * kCWarps;
    const int64_t rows_per_block = (32 / T) * kCWarps;
    const unsigned blocks = (unsigned)((P.n + rows_per_block - 1) / rows_per_block);
    launch_shared(share, forces_contacts_mixed<NEAR, T>, blocks, kCWarps * 32, smem, st, P, S, PV, BV, MX);
}

template <int SL>
void launch_hamaker_all(const Params &P, const PairView &PV, const MixedExtra &MX, cudaStream_t st, int share) {
    const unsigned blocks = (unsigned)((P.n + 31) / 32);
    auto k = P.hamaker_model == LG_HAMAKER_LIMITED      ? forces_hamaker_all<LG_HAMAKER_LIMITED, SL>
             : P.hamaker_model == LG_HAMAKER_SIMPLIFIED ? forces_hamaker_all<LG_HAMAKER_SIMPLIFIED, SL>
                                                        : forces_hamaker_all<LG_HAMAKER_FULL, SL>;
    launch_shared(share, k, blocks, 32 * SL, 0, st, P, PV, MX);
}

template <bool VERLET, int L, int SL>
void launch_hamaker(const Params &P, const PairView &PV, const MixedExtra &MX, cudaStream_t st, int share) {
    const unsigned blocks = (unsigned)((P.n * L + kHThreads - 1) / kHThreads);
    if (P.hamaker_model == LG_HAMAKER_LIMITED)
        launch_shared(share, forces_hamaker_mixed<VERLET, LG_HAMAKER_LIMITED, L, SL>, blocks, kHThreads, 0, st, P, PV, MX);
    else if (P.hamaker_model == LG_HAMAKER_SIMPLIFIED)
        launch_shared(share, forces_hamaker_mixed<VERLET, LG_HAMAKER_SIMPLIFIED, L, SL>, blocks, kHThreads, 0, st, P, PV, MX);
    else
        launch_shared(share, forces_hamaker_mixed<VERLET, LG_HAMAKER_FULL, L, SL>, blocks, kHThreads, 0, st, P, PV, MX);
}

}  // namespace

// Slices per 32-row group of the Hamaker kernel: the most slices that keep the launch within about
// two waves of resident warps (152 SMs x 20); rows of long launches are not sliced.
int mixed_hamaker_slices(int64_t n) {
    if (LG_MIXED_SLICES == 1 || LG_MIXED_SLICES == 2 || LG_MIXED_SLICES == 4 || LG_MIXED_SLICES == 8)
        return LG_MIXED_SLICES;
    const int64_t two_waves = 2 * 152 * 20;
    const int64_t groups = (n + 31) / 32;
    if (groups * 4 <= two_waves) return 4;
    if (groups * 2 <= two_waves) return 2;
    return 1;
}

// Monomers from which all pairs go to forces_hamaker_all. us a step, lanes along a row / lanes on rows, Hamaker pairs
// only: limited form 1400 monomers 25.7 / 32.2, 2048 41.8 / 41.7, 2500 60.9 / 50.7, 4096 128 / 70, 8192 480 / 180;
// full form 2048 42.0 / 45.2, 2500 61.3 / 55.0, 8192 477 / 319. (The kernel before these two, which queued the
// pairs in range in shared memory, took 47, 81 and 275 for the limited form at 2048, 4096 and 8192.)
constexpr int64_t kHamakerAllFrom = 2304;

// All pairs: every row holds n - 1 partners, so small systems slice their rows further (up to 16
// warps per 32-row group) under the same two-wave bound.
static int mixed_hamaker_slices_all_pairs(int64_t n) {
    const int64_t two_waves = 2 * 152 * 20;
    const int64_t groups = (n + 31) / 32;
    for (int sl = 16; sl > 1; sl /= 2)
        if (groups * sl <= two_waves && (n - 1) >= 4 * kWin * sl) return sl;
    return 1;
}

// Rows per block of owned contact candidates (about 1.8 a row in an aggregate, somewhat more than half of
// them touching): a block's candidates are about two per thread of 128, 64 or 32, and its touching pairs
// one per thread. us a step, 32 / 64 / 128 rows, list radius 4.5 r: 2000 monomers 15.2 / 15.5 / 16.1, 4000 15.3 / 15.5 /
// 16.1, 4800 19.8 / 15.7 / 16.4, 8000 20.9 / 16.6 / 17.1, 16000 23.9 / 18.9 / 18.7, 32768 29.1 / 25.0 / 24.7. (From
// 4800 on nearly every SM has a block of one warp beside its Hamaker block; why those then end late is not known.)
int32_t near_block_rows(int64_t n) { return n >= 32768 ? 128 : n > 4096 ? 64 : 32; }

void launch_near_owners(int64_t n, const PairView &PV, const NearScratch &R, cudaStream_t st) {
    const unsigned blocks = (unsigned)((n + R.rb - 1) / R.rb);
    if (blocks) near_owners<<<blocks, 4 * (unsigned)R.rb, 0, st>>>(n, PV, R);  // four lanes per row
}

int launch_forces_compact_mixed(const Params &P, const StateView &S, const PairView &PV, const BondView &BV, double hdt,
                                double dt, int move_facets, bool kick, bool prev_fused, const MixedExtra &MX,
                                cudaStream_t st, const SideStreams &J, int slices, int contact_lanes, NearScratch R) {
    const bool ver = P.pairs == LG_PAIRS_VERLET;
    const int contacts = P.binary_model != LG_BINARY_NONE ? 1 : 0;
    const int hamaker = P.hamaker_model != LG_HAMAKER_NONE ? 1 : 0;
    int kernels = 1;
    const bool unary = P.n_facets > 0 || P.ext_a;
    const unsigned blocks = (unsigned)((P.n + 63) / 64);
    // the contact kernel runs beside the Hamaker kernel, the unary terms beside both; a lone contact kernel
    // needs no second stream
    const bool fork_c = contacts && (hamaker || unary);
    if (!(ver && PV.near_len)) R.rec = nullptr;
    // The kernels of one evaluation ask for one share of shared memory: otherwise those that use none (Hamaker pairs)
    // and those that use some (contacts) cannot be on one SM together, and one stream's kernel waits for the
    // other's to end. Single steps of 8000 listed particles took 40 us as soon as an SM held more than one
    // contact block, and take 29 with one share for all; all pairs of 700 took 39 and take 23. (A share just large
    // enough did not help everywhere: 42 with 64 KB for all pairs of 700; 72 % was 1 to 5 % slower than 44 from
    // 24000 listed monomers on.)
    // The unary terms' kernel is the exception: it is launched first, states no share, and then the SM keeps what its
    // blocks' own use comes to at full occupancy. What can join it there, from the kernels' start and end times: with
    // 0.4 KB a block (its own) mixed_contacts and the Hamaker kernel, not the row-by-row contacts, which wait for it to
    // end, and the Hamaker blocks behind them; with 2 to 6 KB more all of them; with 8 KB more, or with the others'
    // share stated, none. us a step beside the row-by-row contacts, with 0 / 4 KB more: 9000 monomers on a wall 32.3 /
    // 24.7, 4000 31.4 / 31.8, a body force on 9000 24.6 / 22.0, on 16000 25.2 / 23.9. (Beside mixed_contacts: 9000 25.3 /
    // 25.5, 16000 37.3 / 37.6, the restructuring batch 134.6 / 135.3; with the share stated that took 156.)
    const int share = 44;
    if (fork_c || unary) cudaEventRecord(J.fork, st);
    if (unary) {
        cudaStreamWaitEvent(J.unary, J.fork, 0);
        unary_mixed<<<std::min(blocks, (unsigned)kUnaryBlocks), kUnaryThreads, contacts && !R.rec ? 4096 : 0, J.unary>>>(P, S, MX);
        cudaEventRecord(J.unary_join, J.unary);
        ++kernels;
    }
    if (contacts) {
        const cudaStream_t side = fork_c ? J.side : st;
        if (fork_c) cudaStreamWaitEvent(side, J.fork, 0);
        // the FP64 positions are current unless the step before integrated in float-float
        MixedExtra MC = MX;
        MC.x64 = prev_fused ? nullptr : S.x;
        R.lanes = contact_lanes == 1 ? 1 : 2;
        if (R.rec) {
            const unsigned nb = (unsigned)((P.n + R.rb - 1) / R.rb);
            if (R.rb == 128) launch_shared(share, mixed_contacts<128>, nb, 128, 0, side, P, PV, BV, MC, R);
            else if (R.rb == 64) launch_shared(share, mixed_contacts<64>, nb, 64, 0, side, P, PV, BV, MC, R);
            else launch_shared(share, mixed_contacts<32>, nb, 32, 0, side, P, PV, BV, MC, R);
        } else if (ver && PV.near_len && contact_lanes == 1)
            launch_contacts<true, 1>(P, S, PV, BV, MC, side, share);
        else if (ver && PV.near_len)
            launch_contacts<true, kContactLanes>(P, S, PV, BV, MC, side, share);
        else
            launch_contacts<false, 32>(P, S, PV, BV, MC, side, share);
        if (fork_c) cudaEventRecord(J.join, side);
        ++kernels;
    }
    if (hamaker) {
        switch (slices > 0 ? slices : ver ? mixed_hamaker_slices(P.n) : mixed_hamaker_slices_all_pairs(P.n)) {
            case 16:
                if (ver) launch_hamaker<true, 16, 16>(P, PV, MX, st, share);
                else if (P.n >= kHamakerAllFrom) launch_hamaker_all<16>(P, PV, MX, st, share);
                else launch_hamaker<false, 32, 16>(P, PV, MX, st, share);
                break;
            case 8:
                if (ver) launch_hamaker<true, 8, 8>(P, PV, MX, st, share);
                else launch_hamaker<false, 32, 8>(P, PV, MX, st, share);
                break;
            case 4:
                if (ver) launch_hamaker<true, 4, 4>(P, PV, MX, st, share);
                else launch_hamaker<false, 16, 4>(P, PV, MX, st, share);
                break;
            case 2:
                if (ver) launch_hamaker<true, 2, 2>(P, PV, MX, st, share);
                else launch_hamaker<false, 8, 2>(P, PV, MX, st, share);
                break;
            default:
                if (ver) launch_hamaker<true, 1, 1>(P, PV, MX, st, share);
                else launch_hamaker<false, 8, 1>(P, PV, MX, st, share);
        }
        ++kernels;
    }
    if (fork_c) cudaStreamWaitEvent(st, J.join, 0);
    if (unary) cudaStreamWaitEvent(st, J.unary_join, 0);
    // without facets or a body term the completion of a run's steps integrates in float-float; the
    // FP64 completion serves the rest (and a run's last step when the step before was not fused)
    const bool plain = !unary && MX.s32;
    auto split = [](double d) { const float hi = (float)d; return ff{hi, (float)(d - (double)hi)}; };
    if (plain && kick) {
        launch_shared(share, forces_finish_ff<false>, blocks, 64, 0, st, P, S, contacts, hamaker, split(hdt), split(dt), hdt, dt, MX, PV, R);
        return kernels;
    }
    if (plain && prev_fused) {
        launch_shared(share, forces_finish_ff<true>, blocks, 64, 0, st, P, S, contacts, hamaker, split(hdt), split(dt), hdt, dt, MX, PV, R);
        return kernels;
    }
    if (unary)
        launch_shared(share, forces_finish_mixed<true>, blocks, 64, 0, st, P, S, hdt, dt, move_facets, contacts, hamaker, kick ? 1 : 0, MX, PV, R);
    else
        launch_shared(share, forces_finish_mixed<false>, blocks, 64, 0, st, P, S, hdt, dt, 0, contacts, hamaker, kick ? 1 : 0, MX, PV, R);
    return kernels;
}

}  // namespace lg
