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

// a > b for a nonnegative a (NaN: false), compared as integers, off the FP64 pipe; the bound comes from
// above_bound on the host.
__device__ __forceinline__ bool above(double a, int64_t bound) {
    const int64_t ia = __double_as_longlong(a);
    return ia > bound && ia <= 0x7ff0000000000000ll;
}

// c ? a : b as one select instruction. Choosing a pair's constants by its kind with ?: lets the compiler
// branch on the kind and then make one copy of all that follows for bonds and one for contacts; a warp
// holding both kinds would issue both copies.
__device__ __forceinline__ double pick(int c, double a, double b) {
    double r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.f64 %0, %1, %2, p;\n\t}" : "=d"(r) : "d"(a), "d"(b), "r"(c));
    return r;
}
__device__ __forceinline__ int64_t pick(int c, int64_t a, int64_t b) {
    int64_t r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\tselp.b64 %0, %1, %2, p;\n\t}" : "=l"(r) : "l"(a), "l"(b), "r"(c));
    return r;
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
// CULL: skips pairs beyond contact reach before the square root (the pair kernels' queue holds none).
// SPLIT: three consecutive lanes hold the same slot and lane `part` of them evaluates spring `part` (a
// small system waits for one pair's chain of FP64 instructions, and the springs are half of it); `three`
// names the warp's lanes that take part. Lane 0's pa and lane 1's pal are the results.
template <bool FAST = false, bool CONNECTORS = true, bool CULL = true, bool SPLIT = false>
__device__ __forceinline__ void slot_binary_fp64(const Params &P, const StateView &S, const PairView &PV,
                                                 const BondView &BV, int64_t n, int64_t i, int64_t e, int64_t j,
                                                 const d3 xi_, const d3 vi, const d3 wi, d3 &pa, d3 &pal, int part = 0,
                                                 uint32_t three = 0) {
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
    int kind = bonded ? 1 : 0;
    asm volatile("" : "+r"(kind));  // (its value is hidden from the compiler, see pick)
    const double r = pick(kind, P.sinter.r_part, P.contact.r_part);
    const bool apart = CULL && (kind == 0) & above(sqn(dx), P.contact_skip_d2);
    d3 nn = zero3();
    double overlap = 0.0;
    if (!apart) {
        nn = nrmz(dx);
        overlap = 2.0 * r - dot(dx, nn);
    }
    const bool touching = !(apart | ((kind == 0) & (overlap <= 0)));
    if (!touching) {
        if ((fl & kXiLive) && part == 0) {  // reset_springs (contact_force.h:69,99-101)
#pragma unroll 1
            for (int q = 0; q < 9; ++q) PV.xi[q * xs + e] = 0.0;
            PV.flags[e] = fl & ~kXiLive;
        }
        if (!SPLIT) return;  // (split lanes go on together, storing nothing)
    }
    // component c of the pair's springs at store + c * stride
    double *store = reinterpret_cast<double *>(
        pick(kind, reinterpret_cast<int64_t>(BV.xi + be), reinterpret_cast<int64_t>(PV.xi + e)));
    const int64_t stride = pick(kind, (int64_t)BV.bcap * n, xs);
    const bool have = (fl & (kBonded | kXiLive)) != 0;  // springs of a slot that is not live are zero
    const d3 vj = ld4(S.v, j), wj = ld4(S.w, j);
    const double rp = r - overlap / 2.0;
    const d3 v0 = sub(vi, vj);
    const double v_n = -dot(v0, nn);
    const double f_n = pick(kind, P.sinter.k, P.contact.k) * overlap + pick(kind, P.sinter.gamma_n, P.contact.gamma_n) * v_n;
    const d3 nwi = crs(nn, wi), nwj = crs(nn, wj);
    const d3 v_ij = add(add(v0, scl(rp, nwi)), scl(rp, nwj));
    d3 rel = sub(v_ij, scl(dot(v_ij, nn), nn));               // tangential slip
    const d3 v_r = scl(-rp, sub(nwi, nwj));                   // rolling
    const double v_o = r * (dot(nn, wi) - dot(nn, wj));       // torsion, along nn
    const double dt = pick(kind, P.sinter.dt, P.contact.dt);
    d3 force = zero3(), tau = zero3();
    const uint32_t together = __activemask();  // lanes that take the loop with this one
#pragma unroll 1
    for (int q = SPLIT ? part : 0; q < (SPLIT ? part + 1 : 3); ++q) {
        if (SPLIT && q > 0) {
            const d3 vo = scl(v_o, nn);
            rel = mk3(q == 1 ? v_r.x : vo.x, q == 1 ? v_r.y : vo.y, q == 1 ? v_r.z : vo.z);
            store += 3 * q * stride;
        }
        const double kc = q == 0 ? P.contact.k_t : q == 1 ? P.contact.k_r : P.contact.k_o;
        const double kb = q == 0 ? P.sinter.k_t : q == 1 ? P.sinter.k_r : P.sinter.k_o;
        const double gc = q == 0 ? P.contact.gamma_t : q == 1 ? P.contact.gamma_r : P.contact.gamma_o;
        const double gb = q == 0 ? P.sinter.gamma_t : q == 1 ? P.sinter.gamma_r : P.sinter.gamma_o;
        const double kq = pick(kind, kb, kc), gq = pick(kind, gb, gc);
        int free_pair = kind ^ 1;
        asm volatile("" : "+r"(free_pair));
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
        // (the votes keep branches that no lane takes from being issued under a false predicate)
        if (__any_sync(together, free_pair) && free_pair) {  // Coulomb cap
            const double mu = q == 0 ? P.contact.mu_s : q == 1 ? P.contact.mu_r : P.contact.mu_o;
            const double phi = q == 0 ? P.contact.phi_d : q == 1 ? P.contact.phi_r : P.contact.phi_o;
            const double fs = mu * f_n;
            const double f0n = nrm(f);
            const d3 t = f0n > 0.0 ? dvs_t<FAST>(f, f0n) : zero3();
            double cap = fs;
            const bool slide = !(f0n <= fs);
            if (__any_sync(__activemask(), slide) && slide) {
                cap = mu * phi * f_n;
                xi = scl(ddiv(-1.0, kq), add(scl(cap, t), grel));
            }
            f = scl(f0n < cap ? f0n : cap, t);
        }
        if (!SPLIT || touching) {
            store[0] = xi.x;
            store[stride] = xi.y;
            store[2 * stride] = xi.z;
        }
        store += 3 * stride;
        if (q == 0) {
            force = add(scl(f_n, nn), f);
            tau = neg(scl(rp, crs(nn, f)));
            rel = v_r;
        } else {
            const d3 t = scl(r, q == 1 ? crs(nn, f) : f);
            tau = SPLIT ? t : add(tau, t);
            if (!SPLIT) rel = scl(v_o, nn);
        }
    }
    if (SPLIT) {  // lane 1 adds the three torques, in their order
        const int first = (threadIdx.x & 31) - part;
        const d3 t0 = mk3(__shfl_sync(three, tau.x, first), __shfl_sync(three, tau.y, first), __shfl_sync(three, tau.z, first));
        const d3 t1 = mk3(__shfl_sync(three, tau.x, first + 1), __shfl_sync(three, tau.y, first + 1),
                          __shfl_sync(three, tau.z, first + 1));
        const d3 t2 = mk3(__shfl_sync(three, tau.x, first + 2), __shfl_sync(three, tau.y, first + 2),
                          __shfl_sync(three, tau.z, first + 2));
        tau = add(add(t0, t1), t2);
        const d3 top = part == 0 ? force : tau;
        pa = pal = dvs_t<FAST>(top, part == 0 ? pick(kind, P.sinter.mass, P.contact.mass)
                                             : pick(kind, P.sinter.inertia, P.contact.inertia));
        if (!touching) pa = pal = zero3();
        if (part != 0 || !touching) return;
    } else {
        pa = dvs_t<FAST>(force, pick(kind, P.sinter.mass, P.contact.mass));
        pal = dvs_t<FAST>(tau, pick(kind, P.sinter.inertia, P.contact.inertia));
    }
    if (P.binary_model == LG_BINARY_BREAKING_SINTER) {
        const double fn = nrm(force);
        if (bonded && fn > BV.strength[be]) {
            BV.intact[be] = 0;
            PV.flags[e] = fl & ~(kBonded | (0xffu << 8));
        }
    }
    if ((fl & (kBonded | kXiLive)) == 0) PV.flags[e] = fl | kXiLive;
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
    if (hm == LG_HAMAKER_LIMITED && above(d2, P.hamaker_skip_d2)) return ha;
    const double rn = droot(d2);
    if (hm == LG_HAMAKER_LIMITED && above(rn, P.hamaker_cut)) return ha;
    return hamaker_accel_n<FAST>(hm, P.hamaker, P.hc, sub(xj, xi_), rn);
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
