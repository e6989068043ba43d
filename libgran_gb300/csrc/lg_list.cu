// lg_list.cu -- Verlet-list build (sm_103a): bounding box and grid, counting sort by cell, row build with
// spring carry. Compiled with --fmad=false (the list test is the reference's FP64 expression).
//
// What bounds it: launch and dependency latency in the sort's small kernels, instruction issue in the row
// build. Measured for 32768 monomers / a batch of 376,000 in 1024 systems (cold caches), us: sort 37 / 90 -> 26 / 69,
// row build 83 / 987 -> 61 / 296 (80 -> 34 warm). The sort takes four launches instead of nine; a batch's systems
// have grids of their own (one grid over all of them spans the space between, so its cells were three list radii wide and
// held 27 times the candidates); candidates come cell by cell with their positions, one load each, in runs
// cut to the row's reach (94 a row instead of 172); eight lanes build a row instead of 32.
#include <algorithm>

#include "lg_common.cuh"
#include "lg_kernels.h"

namespace lg {

namespace {
constexpr int kBoxThreads = 256;
constexpr int kLineThreads = 256;
// Batch: particles of a system per block of the passes over its grid, one per thread. (With one block per system
// a build grew with the largest: systems of 32768 + 32768 monomers 225 us, 100,000 + 500 508; now 116 and 200, and
// 114 and 200 for one system as large.)
constexpr int kPartRows = 256;
constexpr int kBuildRows = 32;    // rows per block of build_rows
constexpr int kBuildLanes = 8;    // lanes per row
constexpr int kBuildThreads = kBuildRows * kBuildLanes;
constexpr int kBuildAhead = 2;    // candidates per lane whose loads are in flight together
constexpr int kCellsX = 4;        // cells along x per cell width along y and z
constexpr int kLongLine = 1024;   // cells along x above which another axis is considered for the lines
constexpr int kSortBlock = 4;     // partners per lane ranked together
constexpr uint32_t kLive = 0x80000000u;  // staged old partner: its springs are live
constexpr uint32_t kNone = 255u;         // no old slot
}  // namespace

// Order-preserving integer image of a double (FP64 comparisons issue slowly on this GPU); NaN is left out by
// the caller.
__device__ __forceinline__ int64_t key_of(double v) {
    const int64_t b = __double_as_longlong(v);
    return b < 0 ? b ^ 0x7fffffffffffffffll : b;
}
__device__ __forceinline__ double of_key(int64_t k) { return __longlong_as_double(k < 0 ? k ^ 0x7fffffffffffffffll : k); }

struct Box {
    int64_t lo[3], hi[3];
};
__device__ __forceinline__ Box empty_box() {
    const int64_t big = 0x7fffffffffffffffll;
    return Box{{big, big, big}, {-big, -big, -big}};
}
__device__ __forceinline__ void box_add(Box &b, const int64_t (&lo)[3], const int64_t (&hi)[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        b.lo[c] = lo[c] < b.lo[c] ? lo[c] : b.lo[c];
        b.hi[c] = hi[c] > b.hi[c] ? hi[c] : b.hi[c];
    }
}
__device__ __forceinline__ void box_point(Box &b, dbl4 q) {
    const double p[3] = {q.x, q.y, q.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int64_t k = key_of(p[c]);
        if ((uint64_t)(__double_as_longlong(p[c]) << 1) > 0xffe0000000000000ull) continue;  // NaN
        b.lo[c] = k < b.lo[c] ? k : b.lo[c];
        b.hi[c] = k > b.hi[c] ? k : b.hi[c];
    }
}
// the block's box, in thread 0
__device__ __forceinline__ void block_box(Box &b, Box *s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Box u;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            u.lo[c] = __shfl_xor_sync(0xffffffffu, b.lo[c], o);
            u.hi[c] = __shfl_xor_sync(0xffffffffu, b.hi[c], o);
        }
        box_add(b, u.lo, u.hi);
    }
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < (int)blockDim.x / 32; ++w) box_add(b, s[w].lo, s[w].hi);
    __syncthreads();
}

// The grid of one system over its box: cells just above r_verlet wide in y and z (FP32 cell coordinates of
// particles within r_verlet of each other then differ by at most one) and a quarter of that in x, where a
// row's candidates are runs cut to its own reach; all grow by 1.25 until there are at most max_cells. One warp takes a
// line of cells along x (line_starts), so a system that stretches along x and is much thinner elsewhere has its
// lines along its thinnest axis instead (a chain of 20000 along x 258 -> 58 us a build; along z 60): the coordinates of
// the sorted list are then turned, beginning with that axis. Also the FP32 accept / reject bounds of the squared list
// radius for positions stored relative to the grid origin. Returns the number of cells.
__device__ __forceinline__ int32_t grid_of(const Box &b, GridDev *g, double rv, double rnear, int64_t max_cells) {
    double lo[3], hi[3], span = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const bool any = b.lo[c] <= b.hi[c];
        lo[c] = any ? of_key(b.lo[c]) : 0.0;
        hi[c] = any ? of_key(b.hi[c]) : 0.0;
        const double d = hi[c] - lo[c];
        if (d > span) span = d;
    }
    // a coordinate relative to lo rounds to FP32 within span 2^-24, its product with 1 / edge within
    // as much again
    double edge = rv * (1.0 + 1e-5) + 8.0 * span * 1.1920928955078125e-7;
    int32_t turn = 0;
    if (4.0 * (hi[0] - lo[0]) > (double)kLongLine * edge) {
        const int32_t thin = hi[1] - lo[1] < hi[2] - lo[2] ? 1 : 2;
        if (4.0 * (hi[thin] - lo[thin]) < hi[0] - lo[0]) turn = thin;
    }
    int64_t dim[3];
    double cells = 0.0;
    for (int it = 0; it < 4096; ++it) {
        cells = 1.0;
        const xd::Divisor d = xd::divisor(edge);
        for (int c = 0; c < 3; ++c) {
            bool ok = true;
            const int a = turn + c < 3 ? turn + c : turn + c - 3;
            const double ext = c == 0 ? (double)kCellsX * (hi[a] - lo[a]) : hi[a] - lo[a];
            double m = xd::quotient(ext, d, ok);
            if (!ok) m = ext / edge;
            m = floor(m) + 1.0;
            dim[c] = m < 1.0 ? 1 : (int64_t)m;
            cells *= (double)dim[c];
        }
        if (cells <= (double)max_cells) break;
        edge *= 1.25;
    }
    if (!(cells <= (double)max_cells) || !(cells >= 1.0) || !(edge < 1e30)) {  // non-finite or huge: one cell
        dim[0] = dim[1] = dim[2] = 1;
        edge = 1e30;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        g->lo[c] = lo[c];
        g->dim[c] = (int32_t)dim[c];
    }
    g->turn = turn;
    g->edge = (float)edge;
    g->inv_edge = (float)ddiv(1.0, edge);
    // cell boundaries are uncertain by the rounding of the cell coordinates
    const int64_t most = dim[0] > dim[1] ? (dim[0] > dim[2] ? dim[0] : dim[2]) : (dim[1] > dim[2] ? dim[1] : dim[2]);
    g->slack = 1e-3f + (float)most * 2.384185791015625e-7f;
    // FP32 coordinates relative to lo carry an error below span * 2^-24 each; bound |d| by 2 such
    // errors per component and the squared radius by a further relative 1e-6
    const double del = 4.0 * span * 5.9604644775390625e-8 + 1e-300;
    const double lo_r = rv - 2.0 * del, hi_r = rv + 2.0 * del;
    g->rv2_lo = lo_r > 0 ? (float)(lo_r * lo_r * (1.0 - 1e-6)) : 0.0f;
    g->rv2_hi = (float)(hi_r * hi_r * (1.0 + 1e-6));
    g->rn2_hi = rnear > 0 ? (float)((rnear + 2.0 * del) * (rnear + 2.0 * del) * (1.0 + 1e-6)) : -1.0f;
    return (int32_t)(dim[0] * dim[1] * dim[2]);
}

// Leaves the block's box (in thread 0's b) at `at`; true in the block that is the last of `blocks` to do so.
__device__ __forceinline__ bool last_of(const Box &b, Box *at, unsigned *ticket, unsigned blocks, bool *last) {
    if (threadIdx.x == 0) {
        *at = b;
        __threadfence();
        *last = atomicAdd(ticket, 1u) == blocks - 1;
    }
    __syncthreads();
    if (!*last) return false;
    __threadfence();
    return true;
}
// The box over the boxes that `count` blocks left at `part`, in thread 0.
__device__ __forceinline__ void combine_boxes(Box &b, const Box *part, int count, Box *s) {
    b = empty_box();
    for (int q = threadIdx.x; q < count; q += blockDim.x) {
        const long long *p = reinterpret_cast<const long long *>(part + q);
        const int64_t lo[3] = {__ldcg(p), __ldcg(p + 1), __ldcg(p + 2)}, hi[3] = {__ldcg(p + 3), __ldcg(p + 4), __ldcg(p + 5)};
        box_add(b, lo, hi);
    }
    block_box(b, s);
}

// One system: bounding box of the positions, and in the last block to finish the grid. Also zeroes the
// cell counts.
__global__ void __launch_bounds__(kBoxThreads) box_grid(int64_t n, const dbl4 *__restrict__ x, ListScratch L, double rv,
                                                        double rnear, int64_t max_cells) {
    __shared__ Box s[kBoxThreads / 32];
    __shared__ bool last;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t c = t; c < max_cells; c += step) L.count[c] = 0;
    Box b = empty_box();
    for (int64_t i = t; i < n; i += step) box_point(b, x[i]);
    block_box(b, s);
    Box *part = reinterpret_cast<Box *>(L.part);
    if (!last_of(b, part + blockIdx.x, L.ticket, gridDim.x, &last)) return;
    combine_boxes(b, part, (int)gridDim.x, s);
    if (threadIdx.x != 0) return;
    *L.ticket = 0u;
    *L.cursor = 0;
    L.grid->base = 0;
    grid_of(b, L.grid, rv, rnear, max_cells);
}

// A batch: each system has a grid of its own over its active particles (a common grid would have to span the
// empty space between the systems). A system of n_q particles has ceil(n_q / kPartRows) blocks; the last of them
// to finish makes the grid. The systems' cells lie one after another, in any order; a system gets at most
// 8 n_q + 64. Also zeroes the cell counts.
__global__ void __launch_bounds__(kBoxThreads) box_grid_batch(const dbl4 *__restrict__ x, BatchView B, ListScratch L,
                                                              double rv, double rnear, int64_t max_cells) {
    __shared__ Box s[kBoxThreads / 32];
    __shared__ bool last;
    const ListPart w = L.parts[blockIdx.x];
    const int64_t q = w.sys, b0 = B.off[q], b1 = B.off[q + 1];
    for (int64_t c = blockIdx.x * (int64_t)kBoxThreads + threadIdx.x; c < max_cells; c += (int64_t)gridDim.x * kBoxThreads)
        L.count[c] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *L.cursor = 0;
    Box b = empty_box();
    for (int64_t i = b0 + (int64_t)w.part * kBoxThreads + threadIdx.x; i < b1; i += (int64_t)w.parts * kBoxThreads)
        if (!inactive_of(B.hold, i)) box_point(b, x[i]);
    block_box(b, s);
    if (w.parts > 1) {
        if (!last_of(b, reinterpret_cast<Box *>(L.part) + blockIdx.x, L.tickets + q, w.parts, &last)) return;
        combine_boxes(b, reinterpret_cast<Box *>(L.part) + (blockIdx.x - w.part), w.parts, s);
    }
    if (threadIdx.x != 0) return;
    if (w.parts > 1) L.tickets[q] = 0u;
    const int32_t cells = grid_of(b, L.grid + q, rv, rnear, 8 * (b1 - b0) + 64);
    L.grid[q].base = atomicAdd(L.cell_cursor, cells);
}

__device__ __forceinline__ int32_t cell_coord(float f, float inv_edge, int32_t dim) {
    const float u = f * inv_edge;
    const int32_t k = u < 2.0e9f ? (int32_t)u : 2000000000;  // (NaN: the last cell)
    return k < 0 ? 0 : (k >= dim ? dim - 1 : k);
}

__global__ void cell_count(int64_t n, const dbl4 *__restrict__ x, BatchView B, ListScratch L) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i == 0 && B.agg) *L.cell_cursor = 0;  // for the next build
    if (i >= n) return;
    if (inactive_of(B.hold, i)) {  // in no cell: never a candidate of any row
        L.cell_of[i] = -1;
        return;
    }
    const GridDev *g = L.grid + (B.agg ? B.agg[i] : 0);
    const dbl4 q = x[i];
    float4 f = make_float4((float)(q.x - g->lo[0]), (float)(q.y - g->lo[1]), (float)(q.z - g->lo[2]), 0.0f);
    if (g->turn == 1) f = make_float4(f.y, f.z, f.x, 0.0f);
    if (g->turn == 2) f = make_float4(f.z, f.x, f.y, 0.0f);
    const int32_t cx = cell_coord(f.x, (float)kCellsX * g->inv_edge, g->dim[0]), cy = cell_coord(f.y, g->inv_edge, g->dim[1]),
                  cz = cell_coord(f.z, g->inv_edge, g->dim[2]);
    const int32_t c = (cz * g->dim[1] + cy) * g->dim[0] + cx;
    L.cell_of[i] = c;
    L.x32[i] = f;
    atomicAdd(&L.count[g->base + c], 1);
}

// Begin of every cell in the sorted list. Only cells next to each other in x need to be next to each other
// there (a row's candidates are nine runs of cells along x), so the lines of cells along x take their places
// in any order: one warp per line scans its counts and claims the line's length from a cursor. The blocks of
// a system share its lines (one system: all blocks; a batch: those of its parts).
__global__ void __launch_bounds__(kLineThreads) line_starts(ListScratch L, int32_t batch) {
    const ListPart part = batch ? L.parts[blockIdx.x] : ListPart{0, (int32_t)blockIdx.x, (int32_t)gridDim.x};
    const GridDev *g = L.grid + part.sys;
    const int32_t d0 = g->dim[0], lines = g->dim[1] * g->dim[2], base = g->base;
    const int lane = threadIdx.x & 31, warps = part.parts * (kLineThreads / 32);
    for (int32_t w = part.part * (kLineThreads / 32) + (threadIdx.x >> 5); w < lines; w += warps) {
        const int32_t *count = L.count + base + (int64_t)w * d0;
        int32_t *start = L.start + base + (int64_t)w * d0;
        int32_t total = 0;
        for (int32_t c0 = 0; c0 < d0; c0 += 32) total += c0 + lane < d0 ? count[c0 + lane] : 0;
        total = (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)total);
        int32_t at = 0;
        if (lane == 0 && total) at = atomicAdd(L.cursor, total);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int32_t c0 = 0; c0 < d0; c0 += 32) {
            const int32_t v = c0 + lane < d0 ? count[c0 + lane] : 0;
            int32_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (c0 + lane < d0) start[c0 + lane] = at + incl - v;
            at += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
}

// Each particle to its cell's place, with its position (so that a run of candidates is one run of loads); a
// cell's start ends up at its end.
__global__ void cell_scatter(int64_t n, BatchView B, ListScratch L) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t c = L.cell_of[i];
    if (c < 0) return;  // inactive
    const int32_t base = L.grid[B.agg ? B.agg[i] : 0].base;
    float4 f = L.x32[i];
    f.w = __int_as_float((int32_t)i);
    L.sorted[atomicAdd(&L.start[base + c], 1)] = f;
}

// Shared memory of build_rows: 32-row tiles with an odd row stride -- partner, flags, unsorted candidates
// (then near partners), staged old row; old slot and near slot as bytes -- and the rows' bond partners.
__host__ __device__ inline int64_t build_tile_stride(int64_t cap) { return cap | 1; }
__host__ __device__ inline size_t build_smem_bytes(int64_t cap, int64_t bcap) {
    return (size_t)(kBuildRows * build_tile_stride(cap)) * (4 * sizeof(int32_t) + 2) +
           sizeof(int32_t) * (size_t)(kBuildRows * (bcap | 1));
}

// The list test in FP64. Out of line: inlined, its FP64 instructions were issued for every candidate under a
// predicate that is almost always false, and took more than half of the kernel's time (74 -> 34 us).
static __device__ __noinline__ bool listed_exactly(const dbl4 *x, int64_t i, int64_t j, double rv2) {
    return sqn(sub(ld4(x, i), ld4(x, j))) < rv2;
}

// Rows row0 .. row0 + 31: every j != i with squared centre distance < r_verlet^2 (the FP64 test; an FP32
// filter accepts or rejects the clear cases), ascending j, carrying the springs (and live flag) of pairs
// that were already listed, and marking intact bonds.
// Eight lanes per row, four rows per warp (with one row per warp most steps leave lanes idle: about 1560 warp
// instructions a row against about 800): a row's candidates are up to nine runs of consecutive cells, each
// taken kBuildAhead per lane at a time; the accepted ones are appended per row, each with its contact-candidate test in bit 0; each lane ranks its
// partners against the row (they are distinct, so the rank is the slot); the old row, staged in shared
// memory, is searched by bisection; and the block's finished rows are written slot by slot, 32 rows at a
// time.
__global__ void __launch_bounds__(kBuildThreads) build_rows(int64_t n, const dbl4 *__restrict__ x, BatchView B,
                                                            ListScratch L, double rv2, PairView oldv, PairView newv,
                                                            BondView BV, int32_t *err) {
    extern __shared__ int32_t sm[];
    __shared__ int32_t rlen[kBuildRows], rnear[kBuildRows], rold[kBuildRows];
    __shared__ int2 runs[kBuildRows][9];  // the rows' runs of candidates in the sorted list (begin, length)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t cap = newv.cap, ts = build_tile_stride(cap), row0 = (int64_t)blockIdx.x * kBuildRows;
    const int bcap = BV.bcap, bstride = bcap | 1;
    int32_t *tj = sm;
    uint32_t *tf = reinterpret_cast<uint32_t *>(tj + kBuildRows * ts);
    uint32_t *raw = tf + kBuildRows * ts;
    uint32_t *old = raw + kBuildRows * ts;
    int32_t *bond = reinterpret_cast<int32_t *>(old + kBuildRows * ts);
    uint8_t *tp = reinterpret_cast<uint8_t *>(bond + kBuildRows * bstride);
    uint8_t *tnk = tp + kBuildRows * ts;
    const bool near_lists = newv.near_len != nullptr;

    // stage the old rows (partner, live flag) and the intact bonds, slot by slot over the block's rows
    if (tid < kBuildRows) {
        const int64_t i = row0 + tid;
        int32_t o = i < n && oldv.row_len ? oldv.row_len[i] : 0;
        rold[tid] = o > (int32_t)cap ? (int32_t)cap : o;  // both buffers share one capacity
    }
    __syncthreads();
    {
        const int64_t i = row0 + lane;
        const int32_t olen = rold[lane];
        for (int32_t p = warp; p < (int32_t)cap; p += kBuildThreads / 32) {
            if (!__any_sync(0xffffffffu, p < olen)) break;
            if (p < olen) {
                const int64_t e = (int64_t)p * n + i;
                old[lane * ts + p] = (uint32_t)oldv.nbr[e] | ((oldv.flags[e] & kXiLive) ? kLive : 0u);
            }
        }
        for (int b = warp; b < bcap; b += kBuildThreads / 32) {
            int32_t j = -1;
            if (i < n) {
                const int64_t e = (int64_t)b * n + i;
                j = BV.j[e];
                if (j >= 0 && !BV.intact[e]) j = -1;
            }
            bond[lane * bstride + b] = j;
        }
    }

    const int r = tid / kBuildLanes, l = tid % kBuildLanes;
    const uint32_t group = 0xffu << (lane & ~7), below = group & ((1u << lane) - 1u);
    const int64_t i = row0 + r;
    const bool active = i < n && !inactive_of(B.hold, i);  // an inactive particle's row is empty
    float4 fi = make_float4(0.f, 0.f, 0.f, 0.f);
    float rlo = 0.f, rhi = 0.f, rn2 = 0.f;
    if (active) {
        // the row's cell as cell_count placed it, and its nine runs of cells (z, y fixed; x0..x1); a batch's
        // systems have grids of their own, so rows never cross systems
        const GridDev *g = L.grid + (B.agg ? B.agg[i] : 0);
        fi = L.x32[i];
        rlo = g->rv2_lo;
        rhi = g->rv2_hi;
        rn2 = g->rn2_hi;
        const int32_t d0 = g->dim[0], d1 = g->dim[1], d2 = g->dim[2], base = g->base, ci = L.cell_of[i];
        const int32_t cy = (ci / d0) % d1, cz = ci / (d0 * d1);
        const float inv = g->inv_edge, edge = g->edge, slack = g->slack;
        for (int q = l; q < 9; q += kBuildLanes) {
            const int32_t z = cz - 1 + q / 3, y = cy - 1 + q % 3;
            int2 run = make_int2(0, 0);
            if (z >= 0 && z < d2 && y >= 0 && y < d1) {
                // least distances in y and z to that line of cells, and what they leave of the reach in x
                const float ym = fmaxf(edge * (fabsf((float)y + 0.5f - fi.y * inv) - 0.5f - slack), 0.f);
                const float zm = fmaxf(edge * (fabsf((float)z + 0.5f - fi.z * inv) - 0.5f - slack), 0.f);
                const float left = rhi * 1.0001f - ym * ym - zm * zm;
                if (!(left < 0.f)) {
                    const float xr = sqrtf(left) * inv, u = fi.x * inv;
                    const float a = ((float)kCellsX) * (u - xr) - slack, b = ((float)kCellsX) * (u + xr) + slack;
                    const int32_t x0 = a > 0.f ? (a < (float)d0 ? (int32_t)a : d0 - 1) : 0;
                    const int32_t x1 = b > 0.f ? (b < (float)d0 ? (int32_t)b : d0 - 1) : 0;
                    const int32_t c0 = base + (z * d1 + y) * d0;
                    run.x = L.start[c0 + x0] - L.count[c0 + x0];
                    run.y = L.start[c0 + x1] - run.x;
                }
            }
            runs[r][q] = run;
        }
    }
    __syncwarp();
    uint32_t *mine = raw + r * ts;
    int32_t cnt = 0;
    for (int q = 0; q < 9; ++q) {
        const int2 run = active ? runs[r][q] : make_int2(0, 0);
        const int32_t most = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)run.y);
        for (int32_t t0 = 0; t0 < most; t0 += kBuildLanes * kBuildAhead) {
            float4 fb[kBuildAhead];
#pragma unroll
            for (int u = 0; u < kBuildAhead; ++u) {
                const int32_t t = t0 + u * kBuildLanes + l;
                fb[u] = t < run.y ? L.sorted[run.x + t] : make_float4(0.f, 0.f, 0.f, __int_as_float((int32_t)i));
            }
#pragma unroll
            for (int u = 0; u < kBuildAhead; ++u) {
                const int32_t j = __float_as_int(fb[u].w);
                const float ex = fi.x - fb[u].x, ey = fi.y - fb[u].y, ez = fi.z - fb[u].z;
                const float d2f = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
                bool in = j != (int32_t)i && !(d2f > rhi);
                if (in && !(d2f < rlo)) in = listed_exactly(x, i, j, rv2);
                const uint32_t bal = __ballot_sync(0xffffffffu, in) & group;
                if (in) {
                    const int32_t pos = cnt + __popc(bal & below);
                    if (pos < cap) mine[pos] = ((uint32_t)j << 1) | (d2f <= rn2 ? 1u : 0u);
                }
                cnt += __popc(bal);
            }
        }
    }
    if (l == 0) {
        if (cnt > 0) atomicMax(L.max_row, cnt);
        if (cnt > cap) set_error(err, LG_DEVERR_LIST_OVERFLOW);
    }
    if (cnt > cap) cnt = (int32_t)cap;
    __syncwarp();
    // order the row: each lane ranks kSortBlock of its partners at a time against all
    for (int32_t a0 = l; a0 < cnt; a0 += kBuildLanes * kSortBlock) {
        uint32_t v[kSortBlock];
        int32_t rank[kSortBlock];
#pragma unroll
        for (int u = 0; u < kSortBlock; ++u) {
            const int32_t a = a0 + u * kBuildLanes;
            v[u] = a < cnt ? mine[a] : 0u;
            rank[u] = 0;
        }
        for (int32_t t = 0; t < cnt; ++t) {
            const uint32_t w = mine[t];
#pragma unroll
            for (int u = 0; u < kSortBlock; ++u) rank[u] += w < v[u] ? 1 : 0;
        }
#pragma unroll
        for (int u = 0; u < kSortBlock; ++u)
            if (a0 + u * kBuildLanes < cnt) {
                tj[r * ts + rank[u]] = (int32_t)(v[u] >> 1);
                tf[r * ts + rank[u]] = v[u] & 1u;  // the candidate test, until the slot's flags replace it
            }
    }
    __syncthreads();  // (the staged old rows and bonds too)
    int32_t found = 0, intact = 0, nnear = 0;
    const int32_t olen = rold[r];
    for (int b = l; b < bcap; b += kBuildLanes) intact += active && bond[r * bstride + b] >= 0 ? 1 : 0;
    const int32_t longest = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)cnt);
    for (int32_t k0 = 0; k0 < longest; k0 += kBuildLanes) {
        const int32_t k = k0 + l;
        const bool ok = k < cnt;
        uint32_t fl = 0, po = kNone, j = 0;
        bool is_near = false;
        if (ok) {
            j = (uint32_t)tj[r * ts + k];
            // its old slot: mostly the same one, else by bisection
            int32_t lo = k;
            if (!(k < olen && (old[r * ts + k] & ~kLive) == j)) {
                int32_t hi = olen;
                lo = 0;
                while (lo < hi) {
                    const int32_t mid = (lo + hi) >> 1;
                    if ((old[r * ts + mid] & ~kLive) < j)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
            }
            if (lo < olen && old[r * ts + lo] == (j | kLive)) {
                fl = kXiLive;
                po = (uint32_t)lo;
            }
            for (int b = 0; b < bcap; ++b)
                if (bond[r * bstride + b] == (int32_t)j) {
                    fl |= kBonded | ((uint32_t)b << 8);
                    ++found;
                    break;
                }
            if (near_lists) {
                is_near = (fl & kBonded) || tf[r * ts + k] != 0u;
                if (!is_near) {  // apart: its springs reset, so they are not carried
                    fl &= ~kXiLive;
                    po = kNone;
                }
            }
            tf[r * ts + k] = fl;
            tp[r * ts + k] = (uint8_t)po;
        }
        if (near_lists) {
            const uint32_t bal = __ballot_sync(0xffffffffu, is_near) & group;
            if (is_near) {
                const int32_t m = nnear + __popc(bal & below);
                mine[m] = j;
                tnk[r * ts + m] = (uint8_t)k;
            }
            nnear += __popc(bal);
        }
    }
#pragma unroll
    for (int o = kBuildLanes / 2; o > 0; o >>= 1) {
        found += __shfl_xor_sync(0xffffffffu, found, o);
        intact += __shfl_xor_sync(0xffffffffu, intact, o);
    }
    if (l == 0) {
        if (intact != found) set_error(err, LG_DEVERR_BOND_LOST);
        rlen[r] = cnt;
        rnear[r] = nnear;
    }
    __syncthreads();

    // write-out: lane l owns row row0 + l, warp w slots w, w + 8, ...
    const int64_t il = row0 + lane;
    const int32_t len = il < n ? rlen[lane] : 0;
    if (warp == 0 && il < n) newv.row_len[il] = len;
    const int32_t kmax = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)len);
    const int64_t oxs = oldv.cap * n, nxs = newv.cap * n;
    if (near_lists) {
        const int32_t nl = il < n ? rnear[lane] : 0;
        if (warp == 0 && il < n) newv.near_len[il] = nl;
        const int32_t mmax = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)nl);
        for (int32_t m = warp; m < mmax; m += kBuildThreads / 32) {
            if (m >= nl) continue;
            newv.near_j[(int64_t)m * n + il] = (int32_t)raw[lane * ts + m];
            newv.near_k[(int64_t)m * n + il] = tnk[lane * ts + m];
        }
    }
    for (int32_t k = warp; k < kmax; k += kBuildThreads / 32) {
        if (k >= len) continue;
        const int64_t e = (int64_t)k * n + il;
        newv.nbr[e] = tj[lane * ts + k];
        newv.flags[e] = tf[lane * ts + k];
    }
    // the carried springs: the row's eight lanes copy a slot's nine components
    for (int32_t k0 = 0; k0 < longest; k0 += kBuildLanes) {
        const int32_t k = k0 + l;
        uint32_t live = __ballot_sync(0xffffffffu, k < cnt && tp[r * ts + k] != kNone) & group;
        for (; live; live &= live - 1) {
            const int32_t kk = k0 + ((__ffs(live) - 1) & 7);
            const int64_t e = (int64_t)kk * n + i, oe = (int64_t)tp[r * ts + kk] * n + i;
            newv.xi[spring_at(newv.aos, l, e, nxs)] = oldv.xi[spring_at(oldv.aos, l, oe, oxs)];
            if (l == 0) newv.xi[spring_at(newv.aos, 8, e, nxs)] = oldv.xi[spring_at(oldv.aos, 8, oe, oxs)];
        }
    }
}

int64_t list_part_rows() { return kPartRows; }

void launch_list_build(int64_t n, const dbl4 *x, BatchView B, double rv, double r_near, int64_t max_cells,
                       ListScratch &ls, PairView oldv, PairView newv, BondView BV, int32_t *err, cudaStream_t st) {
    const int threads = 256;
    const unsigned blocks = (unsigned)((n + threads - 1) / threads);
    const double rn = newv.near_len ? r_near : 0.0;
    if (B.agg) {
        box_grid_batch<<<(unsigned)ls.nparts, kBoxThreads, 0, st>>>(x, B, ls, rv, rn, max_cells);
    } else {
        // enough blocks for the cell counts to zero, at most the partials' room
        const int64_t want = (std::max<int64_t>(n, max_cells / 4) + kBoxThreads - 1) / kBoxThreads;
        box_grid<<<(unsigned)std::min<int64_t>(want, ls.nparts), kBoxThreads, 0, st>>>(n, x, ls, rv, rn, max_cells);
    }
    cell_count<<<blocks, threads, 0, st>>>(n, x, B, ls);
    const int64_t lb = std::min<int64_t>(std::max<int64_t>(max_cells / 128, 1), 152 * 8);
    line_starts<<<B.agg ? (unsigned)ls.nparts : (unsigned)lb, kLineThreads, 0, st>>>(ls, B.agg ? 1 : 0);
    cell_scatter<<<blocks, threads, 0, st>>>(n, B, ls);
    const size_t smem = build_smem_bytes(newv.cap, BV.bcap);
    static thread_local int attr_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_device != dev) {  // room for the largest capacities (rows and bonds of up to 255 slots)
        cudaFuncSetAttribute(build_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)build_smem_bytes(255, 255));
        attr_device = dev;
    }
    build_rows<<<(unsigned)((n + kBuildRows - 1) / kBuildRows), kBuildThreads, smem, st>>>(n, x, B, ls, rv * rv, oldv,
                                                                                          newv, BV, err);
}

}  // namespace lg
