// lg_list.cu -- Verlet-list build (sm_103a): bounding box and grid, counting sort by cell, row build with
// spring carry. Compiled with --fmad=false (the list test is the reference's FP64 expression).
//
// What bounds it: launch and dependency latency of the sort's small kernels, instruction issue of the
// row build. Measured for 32768 monomers / a batch of 381,000 (us): BUILD_FIGURES
#include <algorithm>

#include "lg_common.cuh"
#include "lg_kernels.h"

namespace lg {

namespace {
constexpr int kBoxThreads = 256;
constexpr int kBuildRows = 32;    // rows per block of build_rows
constexpr int kBuildLanes = 8;    // lanes per row
constexpr int kBuildThreads = kBuildRows * kBuildLanes;
constexpr int kBuildAhead = 3;    // candidates per lane whose loads are in flight together
constexpr int kSortBlock = 4;     // partners per lane ranked together
constexpr uint32_t kLive = 0x80000000u;  // staged old partner: its springs are live
constexpr uint32_t kNone = 255u;         // no old slot
}  // namespace

// Position used for cell hashing: the particle's own coordinates plus, in a batch, the spatial
// offset of its system (systems of a batch keep their own coordinates; the offsets only keep
// their cells apart).
__device__ __forceinline__ dbl4 hash_pos(const dbl4 *__restrict__ x, BatchView B, int64_t i) {
    dbl4 q = x[i];
    if (B.agg) {
        const dbl4 o = B.hoff[B.agg[i]];
        q.x += o.x;
        q.y += o.y;
        q.z += o.z;
    }
    return q;
}

// min and max of three components over the block; the result is valid in thread 0
__device__ __forceinline__ void block_box(double (&lo)[3], double (&hi)[3], double (*s)[kBoxThreads / 32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double a = __shfl_xor_sync(0xffffffffu, lo[c], o), b = __shfl_xor_sync(0xffffffffu, hi[c], o);
            lo[c] = a < lo[c] ? a : lo[c];
            hi[c] = b > hi[c] ? b : hi[c];
        }
        if (lane == 0) {
            s[c][warp] = lo[c];
            s[3 + c][warp] = hi[c];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kBoxThreads / 32; ++w)
            for (int c = 0; c < 3; ++c) {
                if (s[c][w] < lo[c]) lo[c] = s[c][w];
                if (s[3 + c][w] > hi[c]) hi[c] = s[3 + c][w];
            }
    __syncthreads();
}

// Bounding box of the hashed positions, and in the last block to finish the grid: cells of edge just above
// r_verlet (FP32 cell coordinates of particles within r_verlet of each other then differ by at most one);
// the edge grows by 1.25 until the grid has at most max_cells cells. Also fixes the FP32 accept / reject
// bounds of the squared list radius for positions stored relative to the grid origin, and zeroes the
// cell counts.
__global__ void __launch_bounds__(kBoxThreads) box_grid(int64_t n, const dbl4 *__restrict__ x, BatchView B,
                                                        ListScratch L, double rv, double rnear, int64_t max_cells) {
    __shared__ double s[6][kBoxThreads / 32];
    __shared__ bool last;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t c = t; c < max_cells; c += step) L.count[c] = 0;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int64_t i = t; i < n; i += step) {
        const dbl4 q = hash_pos(x, B, i);
        const double p[3] = {q.x, q.y, q.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {  // (a NaN leaves the box alone)
            lo[c] = p[c] < lo[c] ? p[c] : lo[c];
            hi[c] = p[c] > hi[c] ? p[c] : hi[c];
        }
    }
    block_box(lo, hi, s);
    if (threadIdx.x == 0) {
        for (int c = 0; c < 3; ++c) {
            L.part[6 * blockIdx.x + c] = lo[c];
            L.part[6 * blockIdx.x + 3 + c] = hi[c];
        }
        __threadfence();
        last = atomicAdd(L.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = 1e300;
        hi[c] = -1e300;
    }
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double a = __ldcg(L.part + 6 * b + c), z = __ldcg(L.part + 6 * b + 3 + c);
            lo[c] = a < lo[c] ? a : lo[c];
            hi[c] = z > hi[c] ? z : hi[c];
        }
    block_box(lo, hi, s);
    if (threadIdx.x != 0) return;
    *L.ticket = 0u;
    *L.cursor = 0;
    GridDev *g = L.grid;
    double span = 0.0;
    for (int c = 0; c < 3; ++c) {
        const double d = hi[c] - lo[c];
        if (d > span) span = d;
    }
    // a coordinate relative to lo rounds to FP32 within span 2^-24, its product with 1 / edge within
    // as much again
    double edge = rv * (1.0 + 1e-5) + 8.0 * span * 1.1920928955078125e-7;
    int64_t dim[3];
    double cells = 0.0;
    for (int it = 0; it < 4096; ++it) {
        cells = 1.0;
        for (int c = 0; c < 3; ++c) {
            const double m = floor(ddiv(hi[c] - lo[c], edge)) + 1.0;
            dim[c] = m < 1.0 ? 1 : (int64_t)m;
            cells *= (double)dim[c];
        }
        if (cells <= (double)max_cells) break;
        edge *= 1.25;
    }
    if (!(cells <= (double)max_cells) || !(edge < 1e30)) {  // non-finite or huge positions: one cell
        dim[0] = dim[1] = dim[2] = 1;
        edge = 1e30;
    }
    for (int c = 0; c < 3; ++c) {
        g->lo[c] = lo[c];
        g->dim[c] = dim[c];
    }
    g->inv_edge = (float)ddiv(1.0, edge);
    g->ncell = dim[0] * dim[1] * dim[2];
    // FP32 coordinates relative to lo carry an error below span * 2^-24 each; bound |d| by 2 such
    // errors per component and the squared radius by a further relative 1e-6
    const double del = 4.0 * span * 5.9604644775390625e-8 + 1e-300;
    const double lo_r = rv - 2.0 * del, hi_r = rv + 2.0 * del;
    g->rv2_lo = lo_r > 0 ? (float)(lo_r * lo_r * (1.0 - 1e-6)) : 0.0f;
    g->rv2_hi = (float)(hi_r * hi_r * (1.0 + 1e-6));
    g->rn2_hi = rnear > 0 ? (float)((rnear + 2.0 * del) * (rnear + 2.0 * del) * (1.0 + 1e-6)) : -1.0f;
}

__device__ __forceinline__ int32_t cell_coord(float f, float inv_edge, int64_t dim) {
    const float u = f * inv_edge;
    const int32_t k = u < 2.0e9f ? (int32_t)u : 2000000000;  // (NaN converts to 0)
    return k < 0 ? 0 : (k >= (int32_t)dim ? (int32_t)dim - 1 : k);
}

__global__ void cell_count(int64_t n, const dbl4 *__restrict__ x, BatchView B, ListScratch L) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (inactive_of(B.hold, i)) {  // in no cell: never a candidate of any row
        L.cell_of[i] = -1;
        return;
    }
    const GridDev *g = L.grid;
    const dbl4 q = hash_pos(x, B, i);
    const float4 f = make_float4((float)(q.x - g->lo[0]), (float)(q.y - g->lo[1]), (float)(q.z - g->lo[2]), 0.0f);
    const int32_t cx = cell_coord(f.x, g->inv_edge, g->dim[0]), cy = cell_coord(f.y, g->inv_edge, g->dim[1]),
                  cz = cell_coord(f.z, g->inv_edge, g->dim[2]);
    const int32_t c = (cz * (int32_t)g->dim[1] + cy) * (int32_t)g->dim[0] + cx;
    L.cell_of[i] = c;
    L.x32[i] = f;
    atomicAdd(&L.count[c], 1);
}

// Begin of every cell in the sorted list. Only cells next to each other in x need to be next to each other
// there (a row's candidates are nine runs of up to three), so the lines of cells along x take their places
// in any order: one warp per line scans its counts and claims the line's length from a cursor.
__global__ void __launch_bounds__(128) line_starts(ListScratch L) {
    const GridDev *g = L.grid;
    const int64_t d0 = g->dim[0], lines = g->dim[1] * g->dim[2];
    const int lane = threadIdx.x & 31;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < lines;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int32_t *count = L.count + w * d0;
        int32_t *start = L.start + w * d0;
        int32_t total = 0;
        for (int64_t c0 = 0; c0 < d0; c0 += 32) total += c0 + lane < d0 ? count[c0 + lane] : 0;
        total = (int32_t)__reduce_add_sync(0xffffffffu, (unsigned)total);
        int32_t at = 0;
        if (lane == 0 && total) at = atomicAdd(L.cursor, total);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int64_t c0 = 0; c0 < d0; c0 += 32) {
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

// Each particle to its cell's place; a cell's start ends up at its end.
__global__ void cell_scatter(int64_t n, ListScratch L) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t c = L.cell_of[i];
    if (c < 0) return;  // inactive
    L.sorted[atomicAdd(&L.start[c], 1)] = (int32_t)i;
}

// Shared memory of build_rows: 32-row tiles with an odd row stride -- partner, flags, unsorted candidates
// (then near partners), staged old row; old slot and near slot as bytes -- and the rows' bond partners.
__host__ __device__ inline int64_t build_tile_stride(int64_t cap) { return cap | 1; }
__host__ __device__ inline size_t build_smem_bytes(int64_t cap, int64_t bcap) {
    return (size_t)(kBuildRows * build_tile_stride(cap)) * (4 * sizeof(int32_t) + 2) +
           sizeof(int32_t) * (size_t)(kBuildRows * (bcap | 1));
}

// Rows row0 .. row0 + 31: every j != i with squared centre distance < r_verlet^2 (the FP64 test; an FP32
// filter accepts or rejects the clear cases), ascending j, carrying the springs (and live flag) of pairs
// that were already listed, and marking intact bonds.
// Eight lanes per row, four rows per warp (one row per warp spent most of its instructions on steps that
// leave lanes idle: about 1560 warp instructions a row against about 450): the 27 neighbour cells are nine
// runs of consecutive cells, walked as one list of candidates with kBuildAhead per lane in flight; the
// accepted ones are appended per row, each with its contact-candidate test in bit 0; each lane ranks its
// partners against the row (they are distinct, so the rank is the slot); the old row, staged in shared
// memory, is searched by bisection; and the block's finished rows are written slot by slot, 32 rows at a
// time.
__global__ void __launch_bounds__(kBuildThreads) build_rows(int64_t n, const dbl4 *__restrict__ x, BatchView B,
                                                            ListScratch L, double rv2, PairView oldv, PairView newv,
                                                            BondView BV, int32_t *err) {
    extern __shared__ int32_t sm[];
    __shared__ int32_t rlen[kBuildRows], rnear[kBuildRows], rold[kBuildRows];
    __shared__ int32_t rbeg[kBuildRows][9], rpre[kBuildRows][10];  // the runs' begins and their lengths' prefix sums
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
    const GridDev *g = L.grid;

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
    int32_t ai = 0;
    if (active) {
        fi = L.x32[i];
        if (B.agg) ai = B.agg[i];
        // the row's cell as cell_count placed it, and its nine runs of cells (z, y fixed; x0..x1)
        const int32_t d0 = (int32_t)g->dim[0], d1 = (int32_t)g->dim[1], d2 = (int32_t)g->dim[2];
        const int32_t ci = L.cell_of[i];
        const int32_t cx = ci % d0, cy = (ci / d0) % d1, cz = ci / (d0 * d1);
        const int32_t x0 = cx > 0 ? cx - 1 : 0, x1 = cx + 1 < d0 ? cx + 1 : d0 - 1;
        for (int q = l; q < 9; q += kBuildLanes) {
            const int32_t z = cz - 1 + q / 3, y = cy - 1 + q % 3;
            int32_t b = 0, c = 0;
            if (z >= 0 && z < d2 && y >= 0 && y < d1) {
                const int32_t c0 = (z * d1 + y) * d0;
                b = L.start[c0 + x0] - L.count[c0 + x0];
                c = L.start[c0 + x1] - b;
            }
            rbeg[r][q] = b;
            rpre[r][q + 1] = c;
        }
    }
    __syncwarp();
    if (active && l == 0) {
        int32_t run = 0;
        rpre[r][0] = 0;
        for (int q = 1; q < 10; ++q) {
            run += rpre[r][q];
            rpre[r][q] = run;
        }
    }
    __syncwarp();
    const int32_t total = active ? rpre[r][9] : 0;
    const float rlo = g->rv2_lo, rhi = g->rv2_hi, rn2 = g->rn2_hi;
    uint32_t *mine = raw + r * ts;
    int32_t cnt = 0, q = 0;
    const int32_t most = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)total);
    for (int32_t t0 = 0; t0 < most; t0 += kBuildLanes * kBuildAhead) {
        int32_t jb[kBuildAhead];
        float4 fb[kBuildAhead];
        bool same[kBuildAhead];
#pragma unroll
        for (int u = 0; u < kBuildAhead; ++u) {
            const int32_t t = t0 + u * kBuildLanes + l;
            jb[u] = -1;
            if (t < total) {
                while (t >= rpre[r][q + 1]) ++q;
                jb[u] = L.sorted[rbeg[r][q] + (t - rpre[r][q])];
            }
        }
#pragma unroll
        for (int u = 0; u < kBuildAhead; ++u) {
            fb[u] = fi;
            same[u] = true;
            if (jb[u] >= 0) {
                fb[u] = L.x32[jb[u]];
                if (B.agg) same[u] = B.agg[jb[u]] == ai;  // pairs never cross systems
            }
        }
#pragma unroll
        for (int u = 0; u < kBuildAhead; ++u) {
            const int32_t j = jb[u];
            bool in = false;
            const float ex = fi.x - fb[u].x, ey = fi.y - fb[u].y, ez = fi.z - fb[u].z;
            const float d2f = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
            if (j >= 0 && j != (int32_t)i && same[u]) {
                if (d2f < rlo)
                    in = true;
                else if (!(d2f > rhi))
                    in = sqn(sub(ld4(x, i), ld4(x, j))) < rv2;
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, in) & group;
            if (in) {
                const int32_t pos = cnt + __popc(bal & below);
                if (pos < cap) mine[pos] = ((uint32_t)j << 1) | (d2f <= rn2 ? 1u : 0u);
            }
            cnt += __popc(bal);
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
            int32_t lo = 0, hi = olen;
            while (lo < hi) {
                const int32_t mid = (lo + hi) >> 1;
                if ((old[r * ts + mid] & ~kLive) < j)
                    lo = mid + 1;
                else
                    hi = mid;
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
        const uint32_t po = tp[lane * ts + k];
        if (po != kNone) {
            const int64_t oe = (int64_t)po * n + il;
#pragma unroll
            for (int c = 0; c < 9; ++c) newv.xi[spring_at(newv.aos, c, e, nxs)] = oldv.xi[spring_at(oldv.aos, c, oe, oxs)];
        }
    }
}

void launch_list_build(int64_t n, const dbl4 *x, BatchView B, double rv, double r_near, int64_t max_cells,
                       ListScratch &ls, PairView oldv, PairView newv, BondView BV, int32_t *err, cudaStream_t st) {
    const int threads = 256;
    const unsigned blocks = (unsigned)((n + threads - 1) / threads);
    // blocks of the bounding box: enough for the cell counts it zeroes, at most the partials' room
    const int64_t want = (std::max<int64_t>(n, max_cells / 4) + kBoxThreads - 1) / kBoxThreads;
    box_grid<<<(unsigned)std::min<int64_t>(want, ls.nparts), kBoxThreads, 0, st>>>(
        n, x, B, ls, rv, newv.near_len ? r_near : 0.0, max_cells);
    cell_count<<<blocks, threads, 0, st>>>(n, x, B, ls);
    const int64_t warps = std::min<int64_t>(std::max<int64_t>(max_cells / 16, 4), 152 * 64);
    line_starts<<<(unsigned)((warps + 3) / 4), 128, 0, st>>>(ls);
    cell_scatter<<<blocks, threads, 0, st>>>(n, ls);
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
