// lg_pair_fp64.cuh -- the FP64 evaluation of one pair slot and the drift of one particle, shared by the
// row-group kernels (lg_forces_fp64.cu) and the pair kernels (lg_forces_pairs.cu); both compile it with
// --fmad=false.
#pragma once
#include "lg_common.cuh"

namespace lg {

// With connectors (BV.cn): the drift is sinter_step_handler's increment_x then increment_theta
// (sinter_bridge.h:24-42, 55-75): the particle's connectors move with it by dx, then turn by
// dtheta about its moved centre.
// Drift of particle i with kicked velocities vi, wi (stored by the caller).
// A held increment (LG_HOLD_X, LG_HOLD_THETA in `h`) is skipped together with its connector update.
__device__ __forceinline__ void drift_one(int64_t n, int64_t i, dbl4 *__restrict__ x, dbl4 *__restrict__ th, d3 vi,
                                          d3 wi, double dt, const BondView &BV, uint32_t h) {
    const bool hx = h & LG_HOLD_X, hth = h & LG_HOLD_THETA;
    const d3 dx = scl(dt, vi);
    const d3 xn = hx ? ld4(x, i) : add(ld4(x, i), dx);
    if (!hx) st4(x, i, xn);
    const d3 dth = scl(dt, wi);
    if (!hth) st4(th, i, add(ld4(th, i), dth));
    if (BV.cn && !(hx && hth)) {
        const int64_t bs = (int64_t)BV.bcap * n;
        for (int b = 0; b < BV.bcap; ++b) {
            const int64_t e = (int64_t)b * n + i;
            if (BV.j[e] < 0) continue;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                double *cx = BV.cn + (3 * k) * bs + e, *cy = BV.cn + (3 * k + 1) * bs + e, *cz = BV.cn + (3 * k + 2) * bs + e;
                d3 c = mk3(*cx, *cy, *cz);
                if (!hx) c = add(c, dx);
                if (!hth) c = add(c, crs(dth, sub(c, xn)));
                *cx = c.x;
                *cy = c.y;
                *cz = c.z;
            }
        }
    }
}

// a > b for a nonnegative a (or NaN: false): compared as integers, off the FP64 pipe.
__device__ __forceinline__ bool above(double a, double b) {
    const int64_t ia = __double_as_longlong(a), ib = __double_as_longlong(b);
    const int64_t inf = 0x7ff0000000000000ll;
    if (ib < 0 || ib > inf) return a > b;
    return ia > ib && ia <= inf;
}

// The binary functor's value for slot e of row i (P.binary_model != LG_BINARY_NONE); pair state
// (springs, bond state, flags) of slot e is read and written here and nowhere else.
//
// contact_force.h:57-147 and alt_sinter_bridge.h:103-156 / alt_breaking_sinter_bridge.h:89-131 (a bond
// breaks when |f_tot| > strength, :118) share their arithmetic up to the constants and the Coulomb cap,
// so one code path serves both kinds of pair in a warp; the three springs (tangential, rolling,
// torsion) go through one copy of the shear code in a loop, which keeps the kernel small enough for the
// instruction cache (three inlined copies of both functors were fetched once per warp and cost more
// than their arithmetic). The normal keeps the reference's division even in FAST: the overlap 2r - dx.n
// is a small difference of large numbers, so an ulp of n is a large part of it.
template <bool FAST = false, bool CONNECTORS = true>
__device__ __forceinline__ void slot_binary_fp64(const Params &P, const StateView &S, const PairView &PV,
                                                 const BondView &BV, int64_t n, int64_t i, int64_t e, int64_t j,
                                                 const d3 xi_, const d3 vi, const d3 wi, d3 &pa, d3 &pal) {
    const uint32_t fl = PV.flags[e];
    const d3 xj = ld4(S.x, j);
    const d3 dx = sub(xi_, xj);
    pa = zero3();
    pal = zero3();
    const bool bonded = (fl & kBonded) != 0;
    const int64_t be = (int64_t)bond_slot_of(fl) * n + i;
    if (CONNECTORS && bonded && BV.cn) {  // 5-connector model
        const d3 vj = ld4(S.v, j), wj = ld4(S.w, j);
        connector_force(P.connector, P.contact.r_part, P.contact.mass, P.contact.inertia, xi_, xj, vi, vj, wi, wj,
                        BV.cn, (int64_t)BV.bcap * n, be, (int64_t)BV.rev[be] * n + j, pa, pal);
        return;
    }
    const int64_t xs = PV.cap * n;
    const double r = bonded ? P.sinter.r_part : P.contact.r_part;
    bool touching = false;
    d3 nn = zero3();
    double overlap = 0.0;
    if (bonded || !above(sqn(dx), P.contact_skip_d2)) {
        nn = nrmz(dx);
        overlap = 2.0 * r - dot(dx, nn);
        touching = bonded || !(overlap <= 0);
    }
    if (!touching) {
        if (fl & kXiLive) {  // reset_springs (contact_force.h:69,99-101)
#pragma unroll
            for (int q = 0; q < 9; ++q) PV.xi[q * xs + e] = 0.0;
            PV.flags[e] = fl & ~kXiLive;
        }
        return;
    }
    // component c of the pair's springs at store + c * stride
    double *store = bonded ? BV.xi + be : PV.xi + e;
    const int64_t stride = bonded ? (int64_t)BV.bcap * n : xs;
    const bool have = bonded || (fl & kXiLive);  // springs of a slot that is not live are zero
    const d3 vj = ld4(S.v, j), wj = ld4(S.w, j);
    const double rp = r - overlap / 2.0;
    const d3 v0 = sub(vi, vj);
    const double v_n = -dot(v0, nn);
    const double f_n = (bonded ? P.sinter.k : P.contact.k) * overlap + (bonded ? P.sinter.gamma_n : P.contact.gamma_n) * v_n;
    const d3 nwi = crs(nn, wi), nwj = crs(nn, wj);
    const d3 v_ij = add(add(v0, scl(rp, nwi)), scl(rp, nwj));
    d3 rel = sub(v_ij, scl(dot(v_ij, nn), nn));               // tangential slip
    const d3 v_r = scl(-rp, sub(nwi, nwj));                   // rolling
    const double v_o = r * (dot(nn, wi) - dot(nn, wj));       // torsion, along nn
    const double dt = bonded ? P.sinter.dt : P.contact.dt;
    d3 force = zero3(), tau = zero3();
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {
        double kq, gq, mu, phi;
        if (bonded) {
            kq = q == 0 ? P.sinter.k_t : q == 1 ? P.sinter.k_r : P.sinter.k_o;
            gq = q == 0 ? P.sinter.gamma_t : q == 1 ? P.sinter.gamma_r : P.sinter.gamma_o;
            mu = phi = 0.0;
        } else {
            kq = q == 0 ? P.contact.k_t : q == 1 ? P.contact.k_r : P.contact.k_o;
            gq = q == 0 ? P.contact.gamma_t : q == 1 ? P.contact.gamma_r : P.contact.gamma_o;
            mu = q == 0 ? P.contact.mu_s : q == 1 ? P.contact.mu_r : P.contact.mu_o;
            phi = q == 0 ? P.contact.phi_d : q == 1 ? P.contact.phi_r : P.contact.phi_o;
        }
        d3 xi = zero3();
        if (have) xi = mk3(store[0], store[stride], store[2 * stride]);
        // the spring rotated onto the tangent plane, at its length
        d3 xn = sub(xi, scl(dot(xi, nn), nn));
        const double z = sqn(xn);
        if (z > 0.0) {
            xn = dvs_t<FAST>(xn, droot(z));
            xn = scl(nrm(xi), xn);
        }
        const d3 grel = scl(gq, rel);
        d3 f = sub(scl(-kq, xn), grel);
        xi = add(xn, scl(dt, rel));
        if (!bonded) {  // Coulomb cap
            const double fs = mu * f_n, fd = mu * phi * f_n;
            const double f0n = nrm(f);
            const d3 t = f0n > 0.0 ? dvs_t<FAST>(f, f0n) : zero3();
            double cap = fs;
            if (!(f0n <= fs)) {
                xi = scl(ddiv(-1.0, kq), add(scl(fd, t), grel));
                cap = fd;
            }
            f = scl(f0n < cap ? f0n : cap, t);
        }
        store[0] = xi.x;
        store[stride] = xi.y;
        store[2 * stride] = xi.z;
        store += 3 * stride;
        if (q == 0) {
            force = add(scl(f_n, nn), f);
            tau = neg(scl(rp, crs(nn, f)));
            rel = v_r;
        } else {
            tau = add(tau, scl(r, q == 1 ? crs(nn, f) : f));
            rel = scl(v_o, nn);
        }
    }
    if (bonded) {
        if (P.binary_model == LG_BINARY_BREAKING_SINTER && nrm(force) > BV.strength[be]) {
            BV.intact[be] = 0;
            PV.flags[e] = fl & ~(kBonded | (0xffu << 8));
        }
    } else if (!(fl & kXiLive)) {
        PV.flags[e] = fl | kXiLive;
    }
    pa = dvs_t<FAST>(force, bonded ? P.sinter.mass : P.contact.mass);
    pal = dvs_t<FAST>(tau, bonded ? P.sinter.inertia : P.contact.inertia);
}

// The Hamaker term of the pair (i, j) (P.hamaker_model != LG_HAMAKER_NONE).
template <bool FAST = false>
__device__ __forceinline__ d3 slot_hamaker_fp64(const Params &P, const StateView &S, int64_t j, const d3 xi_) {
    const int hm = P.hamaker_model;
    const d3 xj = ld4(S.x, j);
    const d3 dx = sub(xi_, xj);
    d3 ha = zero3();
    // |x_i - x_j| and |x_j - x_i| are the same value (the squares of negated differences are equal)
    const double d2 = sqn(dx);
    if (hm == LG_HAMAKER_LIMITED && d2 > P.hamaker_skip_d2) return ha;
    const double rn = droot(d2);
    if (hm == LG_HAMAKER_LIMITED && rn > P.hamaker.r_cutoff) return ha;
    return hamaker_accel_n<FAST>(hm, P.hamaker, sub(xj, xi_), rn);
}

// The pair value of a slot: binary + Hamaker as the reference's container adds them.
__device__ __forceinline__ void combine_pair_fp64(bool have_binary, bool have_hamaker, const d3 &pb, const d3 &pbl,
                                                  const d3 &ha, d3 &pa, d3 &pal) {
    pa = pb;
    pal = pbl;
    if (have_hamaker) {
        if (have_binary) {
            pa = add(pa, ha);
            pal = add(pal, zero3());
        } else {
            pa = ha;
            pal = zero3();
        }
    }
}

// One slot of row i: the binary functor's pair value plus the Hamaker term, in that order (the
// reference's container returns binary + hamaker for each pair, operator_overloads.h:16-20).
template <bool FAST = false>
__device__ __forceinline__ void slot_pair_fp64(const Params &P, const StateView &S, const PairView &PV,
                                               const BondView &BV, int64_t n, int64_t i, int64_t e, int64_t j,
                                               const d3 xi_, const d3 vi, const d3 wi, d3 &pa_out, d3 &pal_out) {
    const bool hb = P.binary_model != LG_BINARY_NONE, hh = P.hamaker_model != LG_HAMAKER_NONE;
    d3 pb = zero3(), pbl = zero3(), ha = zero3();
    if (hb) slot_binary_fp64<FAST>(P, S, PV, BV, n, i, e, j, xi_, vi, wi, pb, pbl);
    if (hh) ha = slot_hamaker_fp64<FAST>(P, S, j, xi_);
    combine_pair_fp64(hb, hh, pb, pbl, ha, pa_out, pal_out);
}

}  // namespace lg
