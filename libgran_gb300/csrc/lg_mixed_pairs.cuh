// lg_mixed_pairs.cuh -- the per-pair and per-row pieces of the mixed-precision force evaluation,
// shared by the kernels of lg_forces_compact_mixed.cu (contacts and Hamaker on two streams, then a
// completion kernel) and the persistent step kernel of lg_step_mixed.cu (the same rows as work items
// of one launch). Inline device code only: each translation unit compiles it with its own flags
// (both with approximate FP32 division and square root in the pair formulas; the float-float steps
// use explicitly rounded intrinsics).
//
// Precision: positions come as interleaved float-float pairs (MixedExtra::x32, hi + lo = x -
// origin) and a pair's separation and q = |d|^2 - (2r)^2 are formed with error-free FP32
// transformations (separation_ff), so the surface gap and the overlap keep FP32 relative precision
// however small they are; velocities come as float-float copies (MixedExtra::v32); springs are
// float-float pairs in 8-byte slots, one 9-component record per slot or bond (spring_at), updated
// by FP32 increments (shear_ff). A pair's two orders give values that are exactly equal or opposite, so a
// kernel may evaluate either and use it for both. No pair costs an FP64 operation, except the FP64 overlap of a pair
// at the contact threshold (overlap_fp64). Per-row sums are float-float (compensated) FP32
// accumulations in an order fixed by the row alone.
#pragma once
#include <cstddef>

#include "lg_compact.cuh"
#include "lg_kernels.h"

namespace lg {
namespace mixed {

using compact::kWin;

// ---- contact / bond items ----
constexpr int kCRound = 32;  // entries per lane classified per round
constexpr int kCQ = 64;      // contact queue capacity (>= 32 + 31)
#ifndef LG_CONTACT_LANES
#define LG_CONTACT_LANES 2   // lanes per row (compile-time override for tuning)
#endif
constexpr int kContactLanes = LG_CONTACT_LANES;
struct ContactSmem {
    float cres[kCQ][6];  // results: linear and angular acceleration
    float4 chj[kCQ];     // partner's position, high part (read while classifying)
    int32_t cj[kCQ];     // partner
    int32_t ck[kCQ];     // slot in the owner's row
    uint32_t cfl[kCQ];   // the slot's flags (read while classifying)
    uint8_t cown[kCQ];   // owner lane
    uint32_t cball[kCRound];
    int32_t cbase[kCRound];
    float4 xh[32], xl[32];  // the rows' own positions (float-float)
    float4 vh[32], vl[32];  // the rows' own velocities (float-float)
    float4 wh[32];          // the rows' own spins (FP32)
};

struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 fm(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 fadd(f3 a, f3 b) { return fm(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ f3 fsub(f3 a, f3 b) { return fm(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ f3 fscl(float s, f3 a) { return fm(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float fdot(f3 a, f3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ f3 fcrs(f3 a, f3 b) {
    return fm(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// Hamaker factor of hamaker_force.h:36-40 with two reciprocals:
// s = -A/6 [ (4r+2h) u - 2 w - 4 r^2 w^3 - 2 r^2 (4r+2h) u^2 ], u = 1/((4r+h) h), w = 1/(2r+h).
__device__ __forceinline__ float ham_factor(int mode, float A, float r, float h) {
    if (mode == LG_HAMAKER_SIMPLIFIED) return 2.0f * A * r / (h * h);
    float u = 1.0f / ((4.0f * r + h) * h);
    float w = 1.0f / (2.0f * r + h);
    float a = 4.0f * r + 2.0f * h;
    float br = a * u - 2.0f * w - 4.0f * r * r * (w * w * w) - 2.0f * r * r * a * (u * u);
    return -A / 6.0f * br;
}

// Float-float arithmetic (a value is hi + lo with |lo| <= ulp(hi) / 2). The _rn intrinsics keep the
// compiler from contracting or reordering the error-free steps.
struct ff {
    float hi, lo;
};
// TwoSum (Knuth): s + e == a + b exactly, whatever the magnitudes of a and b.
__device__ __forceinline__ ff two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return ff{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
// Compensated accumulation a += b: the rounding error of every addition is kept in a.lo.
__device__ __forceinline__ void ff_acc(ff &a, float b) {
    const ff s = two_sum(a.hi, b);
    a.hi = s.hi;
    a.lo = __fadd_rn(a.lo, s.lo);
}
// a += b for a stored spring component, renormalised so that |lo| <= ulp(hi) / 2 again.
__device__ __forceinline__ void ff_add_norm(ff &a, float b) {
    const ff s = two_sum(a.hi, b);
    const float lo = __fadd_rn(a.lo, s.lo);
    const float hi = __fadd_rn(s.hi, lo);
    a = ff{hi, __fsub_rn(lo, __fsub_rn(hi, s.hi))};
}

// Shear spring (contact_force.h:105-147, Coulomb-capped; alt_sinter_bridge.h:137-156, bond form)
// with the spring vector held as float-float components. Each evaluation computes, in FP32, the
// increment of the spring: the rotation onto the tangent plane, -(xi.n) n, the rescale to the old
// magnitude, (s - 1)(xi - (xi.n) n) with s - 1 evaluated as a series for small tilts, and the
// stretch rel*dt; the increment is small next to xi and is added to the float-float spring, so
// rounding does not accumulate at the spring's own scale. The dynamic (sliding) branch sets the
// spring outright.
__device__ __forceinline__ f3 shear_ff(ff (&xi)[3], f3 n, float stiffness, float damping, float normal_force,
                                       float mu_s, float phi, f3 rel, float dtf, bool coulomb) {
    const f3 xf = fm(xi[0].hi, xi[1].hi, xi[2].hi);  // the FP32 rounding of the spring
    f3 drot = fm(0.f, 0.f, 0.f);
    const float xx = fdot(xf, xf);
    if (xx > 0.0f) {
        const float c = fdot(xf, n);
        const f3 xr = fsub(xf, fscl(c, n));
        const float e = (c * c) / xx;
        float sm1 = 0.0f;
        if (e < 1.0f) sm1 = e < 1e-3f ? e * (0.5f + 0.375f * e) : rsqrtf(1.0f - e) - 1.0f;
        drot = fadd(fscl(-c, n), fscl(sm1, xr));
    }
    const f3 xn = fadd(xf, drot);
    const f3 f0 = fsub(fscl(-stiffness, xn), fscl(damping, rel));
    f3 f = f0;
    bool slide = false;
    if (coulomb) {
        const float fs = mu_s * normal_force;
        const float fd = mu_s * phi * normal_force;
        const float f0n = sqrtf(fdot(f0, f0));
        const f3 t = f0n > 0.0f ? fscl(1.0f / f0n, f0) : fm(0.f, 0.f, 0.f);
        slide = !(f0n <= fs);
        if (slide) {
            const f3 nx = fscl(-1.0f / stiffness, fadd(fscl(fd, t), fscl(damping, rel)));
            xi[0] = ff{nx.x, 0.f};
            xi[1] = ff{nx.y, 0.f};
            xi[2] = ff{nx.z, 0.f};
        }
        f = fscl(fminf(slide ? fd : fs, f0n), t);
    }
    if (!slide) {
        const f3 dxi = fadd(drot, fscl(dtf, rel));
        ff_add_norm(xi[0], dxi.x);
        ff_add_norm(xi[1], dxi.y);
        ff_add_norm(xi[2], dxi.z);
    }
    return f;
}

// Separation d = x_i - x_j (FP32) and q = |d|^2 - (2r)^2 from float-float positions. Per component
// the high parts' difference is split exactly (TwoSum) and its error joins the low parts'
// difference, so dh + dl equals the separation to about 2^-48 of the coordinates. Then
// (dh + dl)^2 = dh^2 + dl (2 dh + dl) with dh^2 split exactly by FMA, the three large squares added
// with TwoSum, and -(2r)^2 (fr_hi + fr_lo) subtracted: that subtraction is exact (Sterbenz) whenever
// |d| is within a factor sqrt(2) of 2r, and otherwise |q| >= 2 r^2, so q keeps FP32 relative
// precision however small the surface gap or the overlap is.
struct SepFF {
    f3 d;
    float q;
};
__device__ __forceinline__ SepFF separation_ff(float4 hi, float4 lo, float4 hj, float4 lj, float fr_hi, float fr_lo) {
    const ff tx = two_sum(hi.x, -hj.x), ty = two_sum(hi.y, -hj.y), tz = two_sum(hi.z, -hj.z);
    const float lx = __fadd_rn(tx.lo, __fsub_rn(lo.x, lj.x));
    const float ly = __fadd_rn(ty.lo, __fsub_rn(lo.y, lj.y));
    const float lz = __fadd_rn(tz.lo, __fsub_rn(lo.z, lj.z));
    const float px = __fmul_rn(tx.hi, tx.hi), py = __fmul_rn(ty.hi, ty.hi), pz = __fmul_rn(tz.hi, tz.hi);
    const float ex = __fmaf_rn(tx.hi, tx.hi, -px), ey = __fmaf_rn(ty.hi, ty.hi, -py), ez = __fmaf_rn(tz.hi, tz.hi, -pz);
    const float cx = lx * (2.0f * tx.hi + lx), cy = ly * (2.0f * ty.hi + ly), cz = lz * (2.0f * tz.hi + lz);
    const ff s1 = two_sum(px, py);
    const ff s2 = two_sum(s1.hi, pz);
    const float s3 = __fsub_rn(s2.hi, fr_hi);
    const float rest = (s1.lo + s2.lo) + ((ex + ey) + ez) + ((cx + cy) + cz) - fr_lo;
    return SepFF{fm(tx.hi + lx, ty.hi + ly, tz.hi + lz), s3 + rest};
}

// c ? a : b as one select instruction (see contact_pair).
__device__ __forceinline__ float pick(int c, float a, float b) {
    float r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.f32 %0, %1, %2, p;\n\t}" : "=f"(r) : "f"(a), "f"(b), "r"(c));
    return r;
}

// One contact or bond pair (contact_force.h:57-147, alt_sinter_bridge.h:103-156) from the two particles'
// float-float positions and velocities and FP32 spins: the force on i, and the three parts of its torque
// (rr n x f_r, rp n x f_t, rr f_o). The springs s (xi_t, xi_r, xi_o) are updated. Returns false, with
// nothing done, when the pair does not touch.
//
// Seen from j (everything swapped) the normal, the slip and the torsion change sign and the rolling
// velocity does not, in every intermediate value and to the last bit (each operation rounds
// symmetrically, and the two rotation terms are added to each other before anything else): the force is
// the negative, xi_t and xi_o are the negatives, xi_r is the same, n x f_r and f_o are the negatives and
// n x f_t is the same. mixed_contacts evaluates a pair once on that ground.
struct Body {
    float4 xh, xl, vh, vl, w;
};
struct ContactOut {
    f3 force, roll, slide, twist;  // force; n x f_r, n x f_t, f_o
    float rr, rp;
};
__device__ __forceinline__ Body body_of(const MixedExtra &M, int64_t n, int64_t i) {
    return Body{M.x32[2 * i], M.x32[2 * i + 1], M.v32[i], M.v32[n + i], M.v32[2 * n + i]};
}
__device__ __forceinline__ f3 torque_of(const f3 &roll, const f3 &slide, const f3 &twist, float rr, float rp) {
    return fadd(fsub(fscl(rr, roll), fscl(rp, slide)), fscl(rr, twist));
}
__device__ __forceinline__ bool contact_pair(const Params &P, const MixedExtra &M, bool bonded, int64_t i, int64_t j,
                                             const Body &bi, const Body &bj, ff (&s)[3][3], ContactOut &o) {
    int kind = bonded ? 1 : 0;
    asm volatile("" : "+r"(kind));  // (its value is hidden from the compiler, see pick)
    const SepFF sp = separation_ff(bi.xh, bi.xl, bj.xh, bj.xl, pick(kind, M.b_fr_hi, M.c_fr_hi),
                                   pick(kind, M.b_fr_lo, M.c_fr_lo));
    const f3 dxf = sp.d;
    const float d2f = fdot(dxf, dxf);
    const float rr = pick(kind, M.b_r, M.c_r);
    const float rsd = rsqrtf(d2f);
    // 2r - |d|, from |d|^2 - (2r)^2 (the product rounds on its own in every kernel: the same bits)
    const float overlap = -sp.q / __fadd_rn(__fmul_rn(d2f, rsd), 2.0f * rr);
    bool touching = bonded || overlap > 0.0f;
    // spheres at the contact distance to within rounding (a seeded aggregate places touching
    // monomers there): the FP64 path's overlap decides whether they touch
    if (!bonded && M.x64 && fabsf(sp.q) <= M.q_marg) touching = overlap_fp64(M.x64, i, j, (double)P.contact.r_part) > 0.0;
    if (!touching) return false;
    const f3 n3 = fscl(rsd, dxf);
    // relative velocity v_i - v_j from the float-float copies (exact high-part difference)
    const ff tx = two_sum(bi.vh.x, -bj.vh.x), ty = two_sum(bi.vh.y, -bj.vh.y), tz = two_sum(bi.vh.z, -bj.vh.z);
    const f3 vij0 = fm(tx.hi + (tx.lo + (bi.vl.x - bj.vl.x)), ty.hi + (ty.lo + (bi.vl.y - bj.vl.y)),
                       tz.hi + (tz.lo + (bi.vl.z - bj.vl.z)));
    const f3 wfi = fm(bi.w.x, bi.w.y, bi.w.z), wfj = fm(bj.w.x, bj.w.y, bj.w.z);
    const float kn = pick(kind, M.b_k, M.c_k), gn = pick(kind, M.b_gn, M.c_gn);
    const float rp = rr - 0.5f * overlap;
    const float v_n = -fdot(vij0, n3);
    const float f_n = kn * overlap + gn * v_n;
    const f3 nwi = fcrs(n3, wfi), nwj = fcrs(n3, wfj);
    const f3 v_ij = fadd(vij0, fscl(rp, fadd(nwi, nwj)));
    const f3 v_t = fsub(v_ij, fscl(fdot(v_ij, n3), n3));
    const f3 v_r = fscl(-rp, fsub(nwi, nwj));
    const f3 v_o = fscl(rr * (fdot(n3, wfi) - fdot(n3, wfj)), n3);
    // (the constants are picked by select instructions: with branches the compiler makes one copy of the
    // shear code for bonds and one for contacts, and a warp with both kinds issues both)
    const float dt = pick(kind, M.b_dt, M.c_dt);
    const f3 f_t = shear_ff(s[0], n3, pick(kind, M.b_kt, M.c_kt), pick(kind, M.b_gt, M.c_gt), f_n, M.c_mus, M.c_phid, v_t, dt, !bonded);
    const f3 f_r = shear_ff(s[1], n3, pick(kind, M.b_kr, M.c_kr), pick(kind, M.b_gr, M.c_gr), f_n, M.c_mur, M.c_phir, v_r, dt, !bonded);
    const f3 f_o = shear_ff(s[2], n3, pick(kind, M.b_ko, M.c_ko), pick(kind, M.b_go, M.c_go), f_n, M.c_muo, M.c_phio, v_o, dt, !bonded);
    o.force = fadd(fscl(f_n, n3), f_t);
    o.roll = fcrs(n3, f_r);
    o.slide = fcrs(n3, f_t);
    o.twist = f_o;
    o.rr = rr;
    o.rp = rp;
    return true;
}

// Entry q of a warp's contact queue (contact_rows): evaluates the pair from the row's side.
__device__ __forceinline__ void contact_item(const Params &P, const PairView &PV, const BondView &BV,
                                             const MixedExtra &M, ContactSmem &W, int q, int64_t row0, int64_t n,
                                             int64_t xs, int64_t bs) {
    const int own = W.cown[q];
    const int64_t io = row0 + own;
    const int64_t e = (int64_t)W.ck[q] * n + io;
    const int32_t j = W.cj[q];
    const uint32_t fl = W.cfl[q];
    const bool bonded = (fl & kBonded) != 0;
    const int64_t base = bonded ? (int64_t)bond_slot_of(fl) * n + io : e, stride = bonded ? bs : xs;
    float2 *store = reinterpret_cast<float2 *>(bonded ? BV.xi : PV.xi);
    const int32_t aos = bonded ? BV.aos : PV.aos;
    // every load the pair may need is issued before any arithmetic (one memory round trip): the
    // partner's low position part, velocities and spin, and the springs of a live slot or bond
    const Body bj{W.chj[q], M.x32[2 * j + 1], M.v32[j], M.v32[n + j], M.v32[2 * n + j]};
    ff s[3][3] = {};  // springs of a slot that is not live are zero
    if (bonded || (fl & kXiLive))
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const float2 v = store[spring_at(aos, c, base, stride)];
            s[c / 3][c % 3] = ff{v.x, v.y};
        }
    const Body bi{W.xh[own], W.xl[own], W.vh[own], W.vl[own], W.wh[own]};
    ContactOut o;
    f3 force = fm(0.f, 0.f, 0.f), torque = fm(0.f, 0.f, 0.f);
    if (contact_pair(P, M, bonded, io, j, bi, bj, s, o)) {
#pragma unroll
        for (int c = 0; c < 9; ++c)
            store[spring_at(aos, c, base, stride)] = make_float2(s[c / 3][c % 3].hi, s[c / 3][c % 3].lo);
        force = o.force;
        torque = torque_of(o.roll, o.slide, o.twist, o.rr, o.rp);
        if (bonded) {
            if (P.binary_model == LG_BINARY_BREAKING_SINTER) {
                const float st = (float)BV.strength[base];
                if (fdot(force, force) > st * st) {
                    BV.intact[base] = 0;
                    PV.flags[e] = fl & ~(kBonded | (0xffu << 8));
                }
            }
        } else if (!(fl & kXiLive)) {
            PV.flags[e] = fl | kXiLive;
        }
    } else if (fl & kXiLive) {
#pragma unroll
        for (int c = 0; c < 9; ++c) PV.xi[spring_at(PV.aos, c, e, xs)] = 0.0;
        PV.flags[e] = fl & ~kXiLive;
    }
    W.cres[q][0] = force.x * M.bin_im;
    W.cres[q][1] = force.y * M.bin_im;
    W.cres[q][2] = force.z * M.bin_im;
    W.cres[q][3] = torque.x * M.bin_iI;
    W.cres[q][4] = torque.y * M.bin_iI;
    W.cres[q][5] = torque.z * M.bin_iI;
}

// The Hamaker acceleration of a row's particle towards one partner (hamaker_force.h:28-44; limited form
// hamaker_force.h:86-93). Its last product and the sums over it round on their own (no fused add), so
// that every kernel that adds these terms gives the same bits.
__device__ __forceinline__ f3 hamaker_pair(int hm, const MixedExtra &M, float4 xh, float4 xl, float4 ph, float4 pl) {
    const SepFF sp = separation_ff(xh, xl, ph, pl, M.h_fr_hi, M.h_fr_lo);
    const f3 dxf = sp.d;
    const float d2f = fdot(dxf, dxf);
    const float rsd = rsqrtf(d2f);
    float h = sp.q / (d2f * rsd + 2.0f * M.h_r);  // |d| - 2r to FP32 precision
    h = fmaxf(h, M.h_h0);
    const float sfac = ham_factor(hm, M.h_A, M.h_r, h) * M.inv_mass_h * rsd;
    if (hm == LG_HAMAKER_LIMITED && sp.q > M.h_qcut) return fm(0.f, 0.f, 0.f);
    return fm(__fmul_rn(-sfac, dxf.x), __fmul_rn(-sfac, dxf.y), __fmul_rn(-sfac, dxf.z));  // along x_j - x_i
}

// Partners of row i in the window of kWin slots from slot k0 on (-1: past the row's end).
template <bool VERLET>
__device__ __forceinline__ void window_partners(const PairView &PV, int64_t n, int64_t i, int32_t len, int32_t k0,
                                                int32_t (&j)[kWin]) {
    const char *row = VERLET ? reinterpret_cast<const char *>(PV.nbr + i) : nullptr;
    const uint32_t pitch = 4u * (uint32_t)n;  // bytes from slot to slot (n <= 2^30)
#pragma unroll
    for (int u = 0; u < kWin; ++u) {
        const int32_t k = k0 + u;
        j[u] = -1;
        if (k < len)
            j[u] = VERLET ? *reinterpret_cast<const int32_t *>(row + (uint64_t)(uint32_t)k * pitch)
                          : (k < (int32_t)i ? k : k + 1);
    }
}

// Sum of a window's Hamaker terms in slot order (FP32; the windows' sums are added with compensation).
// Every slot is evaluated and the ones out of range are left out of the sum: without branches the four
// evaluations overlap. SPARSE: a window without a partner in range of any of the warp's rows is passed over.
template <int HM, bool SPARSE = false>
__device__ __forceinline__ f3 window_sum(const MixedExtra &MX, float4 xh, float4 xl, const int32_t (&j)[kWin]) {
    float4 ph[kWin], pl[kWin];
#pragma unroll
    for (int u = 0; u < kWin; ++u) {
        ph[u] = xh;
        pl[u] = xl;
        if (j[u] >= 0) {
            const float4 *p = MX.x32 + 2 * (int64_t)j[u];
            ph[u] = p[0];
            pl[u] = p[1];
        }
    }
    f3 sum = fm(0.f, 0.f, 0.f);
    if (SPARSE) {
        bool any = false;
#pragma unroll
        for (int u = 0; u < kWin; ++u) {
            const float dx = xh.x - ph[u].x, dy = xh.y - ph[u].y, dz = xh.z - ph[u].z;
            any = any || (j[u] >= 0 && fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= MX.near2);
        }
        if (!__any_sync(__activemask(), any)) return sum;
    }
#pragma unroll
    for (int u = 0; u < kWin; ++u) {
        bool on = j[u] >= 0;
        if (HM == LG_HAMAKER_LIMITED) {
            const float dx = xh.x - ph[u].x, dy = xh.y - ph[u].y, dz = xh.z - ph[u].z;
            on = on && fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= MX.near2;
        }
        const f3 a = hamaker_pair(HM, MX, xh, xl, ph[u], pl[u]);
        sum = fm(on ? __fadd_rn(sum.x, a.x) : sum.x, on ? __fadd_rn(sum.y, a.y) : sum.y,
                 on ? __fadd_rn(sum.z, a.z) : sum.z);
    }
    return sum;
}
__device__ __forceinline__ f3 window_sum(int hm, const MixedExtra &MX, float4 xh, float4 xl, const int32_t (&j)[kWin]) {
    if (hm == LG_HAMAKER_LIMITED) return window_sum<LG_HAMAKER_LIMITED>(MX, xh, xl, j);
    if (hm == LG_HAMAKER_SIMPLIFIED) return window_sum<LG_HAMAKER_SIMPLIFIED>(MX, xh, xl, j);
    return window_sum<LG_HAMAKER_FULL>(MX, xh, xl, j);
}

// Float-float sum and product (the product's rounding error from an FMA; results renormalised).
__device__ __forceinline__ ff ff_add(ff a, ff b) {
    const ff s = two_sum(a.hi, b.hi);
    return two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
    const float p = __fmul_rn(a.hi, b.hi);
    const float e = __fmaf_rn(a.hi, b.hi, -p);
    return two_sum(p, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, e)));
}
__device__ __forceinline__ double ff_to_d(ff a) { return (double)a.hi + (double)a.lo; }


// Contact and bond pairs of rows row0 .. row0 + 32/T - 1 (one warp): T lanes per row, lane t of a
// row taking its entries t, t + T, ... (so short candidate lists still fill the warp); each lane folds
// its pairs in entry order and the row's T partial sums are combined in lane order. csum receives the
// contact part of the row's accelerations as float-float pairs.
template <bool NEAR, int T>
__device__ __forceinline__ void contact_rows(const Params &P, const PairView &PV, const BondView &BV,
                                             const MixedExtra &MX, ContactSmem &W, int64_t row0, int lane) {
    const int r = lane / T, sub = lane % T;  // local row and sub-lane
    const int64_t n = P.n;
    const int64_t i = row0 + r;
    const bool active = i < n;
    const uint32_t lt = (1u << lane) - 1u;
    int64_t len = 0;
    float4 hi_i = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
        len = NEAR ? (int64_t)PV.near_len[i] : n - 1;
        hi_i = MX.x32[2 * i];
    }
    if (sub == 0) {
        const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
        W.xh[r] = hi_i;
        W.xl[r] = active ? MX.x32[2 * i + 1] : z4;
        W.vh[r] = active ? MX.v32[i] : z4;
        W.vl[r] = active ? MX.v32[n + i] : z4;
        W.wh[r] = active ? MX.v32[2 * n + i] : z4;
    }
    // iterations: the lane's entries sub, sub + T, ... below len
    const int64_t my_it = len > sub ? (len - sub + T - 1) / T : 0;
    const int64_t itmax = (int64_t)__reduce_max_sync(0xffffffffu, (unsigned)my_it);
    const int64_t xs = PV.cap * n;
    const int64_t bs = (int64_t)BV.bcap * n;
    ff acc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}}, accw[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    __syncwarp();

    // entry of iteration it: partner and slot (-1: none). Candidate lists are loaded two iterations ahead, and
    // their entries' flags and partner positions one iteration ahead of the classification; with all pairs,
    // where the partner follows from the slot, kDeep iterations of flags and positions are in flight (contacts
    // alone, us a step with 1 / 2 / 4: 256 monomers 11.6 / 11.4 / 12.0, 2048 36.7 / 35.9 / 47.6, 8192 776 / 736 / 860;
    // four take more registers than there are).
    constexpr int kDeep = NEAR ? 1 : 2;
    int32_t jn = -1, kn = 0;
    auto load_entry = [&](int64_t it) {
        const int64_t m = it * T + sub;
        jn = -1;
        if (m < len) {
            if (NEAR) {
                jn = PV.near_j[m * n + i];
                kn = PV.near_k[m * n + i];
            } else {
                kn = (int32_t)m;
                jn = (int32_t)(m < i ? m : m + 1);
            }
        }
    };
    int32_t jc = -1, kc = 0;  // the entry being classified (candidate lists), the flags and partner positions ahead
    uint32_t flc[kDeep];
    float4 pjc[kDeep];
    auto take_entry = [&](int d) {  // the loaded entry becomes entry d; its data is requested
        jc = jn;
        kc = kn;
        flc[d] = 0;
        pjc[d] = hi_i;
        if (jn >= 0) {
            flc[d] = PV.flags[(int64_t)kn * n + i];
            pjc[d] = MX.x32[2 * jn];
        }
    };
#pragma unroll
    for (int d = 0; d < kDeep; ++d) {
        load_entry(d);
        take_entry(d);
    }
    if (NEAR) load_entry(1);
    for (int64_t it0 = 0; it0 < itmax;) {
        int ccount = 0, cdone = 0;
        int64_t it = it0;
        for (;;) {
            const bool take = it < itmax && it - it0 < kCRound && ccount + 32 <= kCQ;
            if (take) {
                int32_t j = jc, k = kc;
                if (!NEAR) {
                    k = (int32_t)(it * T) + sub;
                    j = k < len ? (k < i ? k : k + 1) : -1;
                }
                const uint32_t fl = flc[0];
                const float4 pj = pjc[0];
#pragma unroll
                for (int d = 0; d + 1 < kDeep; ++d) {
                    flc[d] = flc[d + 1];
                    pjc[d] = pjc[d + 1];
                }
                if (NEAR) {
                    take_entry(0);
                    load_entry(it + 2);
                } else if (it + kDeep < itmax) {
                    load_entry(it + kDeep);
                    take_entry(kDeep - 1);
                }
                bool cb = false;
                if (j >= 0) {
                    const float dx = hi_i.x - pj.x, dy = hi_i.y - pj.y, dz = hi_i.z - pj.z;
                    if ((fl & kBonded) || fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= MX.contact2f) {
                        cb = true;
                    } else if (fl & kXiLive) {  // reset_springs (contact_force.h:69,99-101)
                        const int64_t e = (int64_t)k * n + i;
#pragma unroll
                        for (int c = 0; c < 9; ++c) PV.xi[spring_at(PV.aos, c, e, xs)] = 0.0;
                        PV.flags[e] = fl & ~kXiLive;
                    }
                }
                const uint32_t bc = __ballot_sync(0xffffffffu, cb);
                if (cb) {
                    const int q = ccount + __popc(bc & lt);
                    W.cj[q] = j;
                    W.ck[q] = k;
                    W.cfl[q] = fl;
                    W.chj[q] = pj;
                    W.cown[q] = (uint8_t)r;
                }
                if (lane == 0) {
                    W.cball[it - it0] = bc;
                    W.cbase[it - it0] = ccount;
                }
                ccount += __popc(bc);
                ++it;
            }
            __syncwarp();
            // full batches of 32 while the round is open, the rest when it closes
            while (ccount - cdone >= 32 || (!take && cdone < ccount)) {
                if (cdone + lane < ccount) contact_item(P, PV, BV, MX, W, cdone + lane, row0, n, xs, bs);
                cdone += 32;
                __syncwarp();
            }
            if (!take) break;
        }
        // the round's pairs, in entry order
        for (int off = 0; off < (int)(it - it0); ++off) {
            const uint32_t bc = W.cball[off];
            if ((bc >> lane) & 1u) {
                const int q = W.cbase[off] + __popc(bc & lt);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    ff_acc(acc[c], W.cres[q][c]);
                    ff_acc(accw[c], W.cres[q][3 + c]);
                }
            }
        }
        __syncwarp();
        it0 = it;
    }
    if (T > 1) {  // the row's partial sums, in lane order, onto its first lane
        const int base = lane - sub;
        // a lane without a touching pair adds zeros, which change nothing: with a warp per row such lanes, nearly
        // all of them, are passed over
        uint32_t some = 0xffffffffu;
        if (T == 32) {
            bool any = false;
#pragma unroll
            for (int c = 0; c < 3; ++c) any = any || acc[c].hi != 0.f || acc[c].lo != 0.f || accw[c].hi != 0.f || accw[c].lo != 0.f;
            some = __ballot_sync(0xffffffffu, any);
        }
#pragma unroll(T == 32 ? 1 : T)
        for (int t = 1; t < T; ++t) {
            if (T == 32) {
                t = __ffs(some & (0xffffffffu << t)) - 1;
                if (t < 0) break;
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float ah = __shfl_sync(0xffffffffu, acc[c].hi, base + t);
                const float al = __shfl_sync(0xffffffffu, acc[c].lo, base + t);
                const float wh = __shfl_sync(0xffffffffu, accw[c].hi, base + t);
                const float wl = __shfl_sync(0xffffffffu, accw[c].lo, base + t);
                if (sub == 0) {
                    ff_acc(acc[c], ah);
                    ff_acc(acc[c], al);
                    ff_acc(accw[c], wh);
                    ff_acc(accw[c], wl);
                }
            }
        }
    }
    if (!active || sub != 0) return;
    MX.csum[3 * i] = make_float4(acc[0].hi, acc[0].lo, acc[1].hi, acc[1].lo);
    MX.csum[3 * i + 1] = make_float4(acc[2].hi, acc[2].lo, accw[0].hi, accw[0].lo);
    MX.csum[3 * i + 2] = make_float4(accw[1].hi, accw[1].lo, accw[2].hi, accw[2].lo);
}

// Hamaker pairs of row row0 + lane, slice sl of kSlices: the windows sl, sl + kSlices, ... acch receives
// the row's partial sum (float-float). HM: the Hamaker form (negative: from P), SPARSE: as window_sum.
template <bool VERLET, int HM = -1, bool SPARSE = false>
__device__ __forceinline__ void hamaker_rows(const Params &P, const PairView &PV, const MixedExtra &MX, int64_t row0,
                                             int sl, int kSlices, int lane, ff (&acch)[3]) {
    const int64_t n = P.n, i = row0 + lane;
    acch[0] = acch[1] = acch[2] = ff{0.f, 0.f};
    if (i >= n) return;
    const int32_t len = VERLET ? PV.row_len[i] : (int32_t)(n - 1);
    const float4 xh = MX.x32[2 * i], xl = MX.x32[2 * i + 1];
    for (int32_t k0 = sl * kWin; k0 < len; k0 += kSlices * kWin) {
        int32_t j[kWin];
        window_partners<VERLET>(PV, n, i, len, k0, j);
        f3 w;
        if constexpr (HM >= 0) w = window_sum<HM, SPARSE>(MX, xh, xl, j);
        else w = window_sum(P.hamaker_model, MX, xh, xl, j);
        ff_acc(acch[0], w.x);
        ff_acc(acch[1], w.y);
        ff_acc(acch[2], w.z);
    }
}

// The completion of a step of a run for a particle that no step handler holds (the body of
// forces_finish_ff below): a, al are the row's float-float accelerations (contact + Hamaker). The
// float-float state is read from MX (x32, v32, s32) and the next step's positions and velocities are
// written to x32o / v32o (MX.x32 / MX.v32 themselves, or the other buffers of a double-buffered
// state); every load of the row precedes its stores.
template <bool LAST>
__device__ __forceinline__ void finish_ff_plain(const StateView &S, int64_t i, int64_t n, ff (&a)[3], const ff (&al)[3],
                                                ff hdt, ff dt, const MixedExtra &MX, float4 *x32o, float4 *v32o) {
    const float4 vh = MX.v32[i], vl = MX.v32[n + i], wh = MX.v32[2 * n + i], wl = MX.s32[i];
    const float4 dh = MX.s32[n + i], dl = MX.s32[2 * n + i], rh = MX.s32[3 * n + i], rl = MX.s32[4 * n + i];
    bool finite = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) finite = finite && isfinite(a[c].hi) && isfinite(al[c].hi);
    if (!finite) set_error(S.err, LG_DEVERR_NONFINITE);
    ff v[3] = {{vh.x, vl.x}, {vh.y, vl.y}, {vh.z, vl.z}};
    ff w[3] = {{wh.x, wl.x}, {wh.y, wl.y}, {wh.z, wl.z}};
    ff dx[3] = {{dh.x, dl.x}, {dh.y, dl.y}, {dh.z, dl.z}};
    ff dr[3] = {{rh.x, rl.x}, {rh.y, rl.y}, {rh.z, rl.z}};
    // end-of-step half kick
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[c] = ff_add(v[c], ff_mul(hdt, a[c]));
        w[c] = ff_add(w[c], ff_mul(hdt, al[c]));
    }
    if (LAST) {
        const d3 x0 = ld4(S.x, i), t0 = ld4(S.th, i);
        st4(S.a, i, mk3(ff_to_d(a[0]), ff_to_d(a[1]), ff_to_d(a[2])));
        st4(S.al, i, mk3(ff_to_d(al[0]), ff_to_d(al[1]), ff_to_d(al[2])));
        st4(S.v_out, i, mk3(ff_to_d(v[0]), ff_to_d(v[1]), ff_to_d(v[2])));
        st4(S.w_out, i, mk3(ff_to_d(w[0]), ff_to_d(w[1]), ff_to_d(w[2])));
        st4(S.x, i, mk3(x0.x + ff_to_d(dx[0]), x0.y + ff_to_d(dx[1]), x0.z + ff_to_d(dx[2])));
        st4(S.th, i, mk3(t0.x + ff_to_d(dr[0]), t0.y + ff_to_d(dr[1]), t0.z + ff_to_d(dr[2])));
        return;
    }
    // the next step's opening half kick and drift
    const float4 xh = MX.x32[2 * i], xl = MX.x32[2 * i + 1];  // loaded before anything is stored
    ff x[3] = {{xh.x, xl.x}, {xh.y, xl.y}, {xh.z, xl.z}};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[c] = ff_add(v[c], ff_mul(hdt, a[c]));
        w[c] = ff_add(w[c], ff_mul(hdt, al[c]));
        const ff step = ff_mul(dt, v[c]);
        x[c] = ff_add(x[c], step);
        dx[c] = ff_add(dx[c], step);
        dr[c] = ff_add(dr[c], ff_mul(dt, w[c]));
    }
    x32o[2 * i] = make_float4(x[0].hi, x[1].hi, x[2].hi, 0.f);
    x32o[2 * i + 1] = make_float4(x[0].lo, x[1].lo, x[2].lo, 0.f);
    v32o[i] = make_float4(v[0].hi, v[1].hi, v[2].hi, 0.f);
    v32o[n + i] = make_float4(v[0].lo, v[1].lo, v[2].lo, 0.f);
    v32o[2 * n + i] = make_float4(w[0].hi, w[1].hi, w[2].hi, 0.f);
    MX.s32[i] = make_float4(w[0].lo, w[1].lo, w[2].lo, 0.f);
    MX.s32[n + i] = make_float4(dx[0].hi, dx[1].hi, dx[2].hi, 0.f);
    MX.s32[2 * n + i] = make_float4(dx[0].lo, dx[1].lo, dx[2].lo, 0.f);
    MX.s32[3 * n + i] = make_float4(dr[0].hi, dr[1].hi, dr[2].hi, 0.f);
    MX.s32[4 * n + i] = make_float4(dr[0].lo, dr[1].lo, dr[2].lo, 0.f);
}

}  // namespace mixed
}  // namespace lg
