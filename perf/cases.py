"""The work that users of libgran_gb300 have it do, as cases to time.

A case is one output interval of a simulation: a driver advances its system by some steps through the
public API and reads the state back (positions, velocities, orientations, spins), as libgran's own
drivers do between two dumps. Every case names its functor set, precision, pair enumeration and
sizes; the systems are seeded random-sequential-attachment aggregates of 14 nm monomers with the
material constants of libgran_gb300.configs.Material.

  listed()           the cases that are timed by name
  draw(rng)          one more case of the same ranges
  prepare(c, seed)   the system (or server) that a driver holds, built from seeded inputs
  run(state)         one output interval through the public API
  exact(c, seed)     what run() returns, from a plain FP64 evaluation of the force laws in torch
  work(c)            bytes and operations of one interval
"""
import math

import numpy as np
import torch

VMAX = 0.1        # m/s, initial velocity components
REBUILD = 20      # steps between Verlet-list rebuilds (libgran's hamaker_neighbor driver)
V_WALL = 1.0      # m/s, moving wall of the restructuring workload
STRENGTH = 1e-8   # N, neck strength of the breaking bonds


# ------------------------------------------------------------------------------------------------
# Cases
# ------------------------------------------------------------------------------------------------
def _case(name, model, ham, precision, n, steps, *, pairs="verlet", count=1, lo=0, hi=0, calls=1, wall=False,
          obs=False, serve=False, sizes_seed=2):
    """n: monomers of a single system, or the median size of a batch's aggregates; count: aggregates;
    lo, hi: size range of a batch (log-normal about n, or log-uniform when n is 0); steps: steps per
    lg_step call; calls: calls per interval; wall: a moving wall facet; obs: the driver also reads
    kinetic observables; serve: the aggregates are requests to the serving loop;
    sizes_seed: seed of a batch's sizes (the inputs' seed draws everything else)."""
    return dict(name=name, model=model, ham=ham, precision=precision, n=n, steps=steps, pairs=pairs, count=count,
                lo=lo, hi=hi, calls=calls, wall=wall, obs=obs, serve=serve, sizes_seed=sizes_seed)


def listed():
    return [
        # libgran's small known-answer drivers: a few dozen particles, every pair, one do_step per
        # call (the drop-in granular_system::do_step), where launches and latency count
        _case("small-40-fp64-do_step", "contact", "full", "fp64", 40, 1, pairs="all", calls=50),
        # the CPU-runnable aggregate of libgran: 256 sintered monomers, every pair, full Hamaker
        _case("aggregate-256-fp64", "sinter", "full", "fp64", 256, 100, pairs="all"),
        # the same in mixed precision
        _case("aggregate-256-mixed", "sinter", "full", "mixed", 256, 200, pairs="all"),
        # a mid-size frictional packing without van der Waals forces, stepped one do_step at a time
        _case("contact-1999-mixed-do_step", "contact", "none", "mixed", 1999, 1, calls=40),
        # a mid-size aggregate whose bonds can break, in FP64 (odd size, Verlet list)
        _case("breaking-5003-fp64", "breaking", "limited", "fp64", 5003, 20),
        # the single large aggregate (contact + limited Hamaker, Verlet list 4.5 r), mixed precision,
        # with the kinetic observables that drivers print at each dump
        _case("aggregate-32768-mixed", "contact", "limited", "mixed", 32768, 40, obs=True),
        # the same in FP64 (libgran's results bit for bit)
        _case("aggregate-32768-fp64", "contact", "limited", "fp64", 32768, 20, obs=True),
        # a parameter study: a thousand independent aggregates of 32 to 2048 monomers in one handle
        _case("batch-1024-mixed", "sinter", "limited", "mixed", 256, 20, count=1024, lo=32, hi=2048),
        # a smaller study in FP64
        _case("batch-96-fp64", "sinter", "limited", "fp64", 256, 20, count=96, lo=32, hi=2048),
        # restructuring: aggregates of 128 to 4096 monomers with breaking bonds on a moving wall
        _case("restructuring-128-wall-mixed", "breaking", "limited", "mixed", 0, 20, count=128, lo=128, hi=4096,
              wall=True),
        # the serving loop: two dozen requests of 64 to 1024 monomers, 100 steps each
        _case("serving-24-mixed", "sinter", "limited", "mixed", 0, 100, count=24, lo=64, hi=1024, serve=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: any functor set and precision, sizes log-uniform."""
    model = rng.choice(["contact", "sinter", "breaking"])
    prec = rng.choice(["fp64", "mixed", "mixed"])
    kind = rng.choice(["all", "verlet", "verlet", "large", "batch", "wall", "serve"])
    if kind == "all":
        n = _log(rng, 9, 700)
        one = rng.random() < 0.4
        c = _case(None, model, rng.choice(["full", "limited", "none"]), prec, n, 1 if one else _log(rng, 10, 100),
                  pairs="all", calls=_log(rng, 10, 50) if one else 1, obs=rng.random() < 0.3)
    elif kind == "verlet":
        one = rng.random() < 0.3
        c = _case(None, model, rng.choice(["limited", "limited", "none"]), prec, _log(rng, 100, 12000),
                  1 if one else _log(rng, 10, 60), calls=_log(rng, 10, 40) if one else 1, obs=rng.random() < 0.3)
    elif kind == "large":
        c = _case(None, model, "limited", prec, _log(rng, 12000, 40000), rng.choice([10, 20, 20, 40]),
                  obs=rng.random() < 0.5)
    elif kind == "batch":
        fp = prec == "fp64"
        c = _case(None, model, "limited", prec, 256, rng.choice([10, 20]), count=_log(rng, 16, 100 if fp else 1000),
                  lo=32, hi=2048)
    elif kind == "wall":
        fp = prec == "fp64"
        c = _case(None, model, "limited", prec, 0, rng.choice([10, 20]), count=_log(rng, 8, 24 if fp else 128),
                  lo=128, hi=4096, wall=True)
    else:
        c = _case(None, "sinter", "limited", prec, 0, 20 * rng.randint(2, 6), count=_log(rng, 6, 24), lo=64, hi=1024,
                  serve=True)
    del c["name"]
    if c["count"] > 1:
        c["sizes_seed"] = rng.randrange(1 << 20)
    return c


# ------------------------------------------------------------------------------------------------
# Inputs (host arrays, as libgran's drivers hold them)
# ------------------------------------------------------------------------------------------------
def _batched(case):
    return case["serve"] or case["count"] > 1 or case["wall"]


def _sizes(case):
    from libgran_gb300 import configs as K
    if not _batched(case):
        return np.array([case["n"]], dtype=np.int64)
    if case["n"]:
        return K.lognormal_sizes(case["count"], case["n"], case["lo"], case["hi"], seed=case["sizes_seed"])
    return K.loguniform_sizes(case["count"], case["lo"], case["hi"], seed=case["sizes_seed"])


def _inputs(case, seed):
    """Sizes, positions, velocities and spins: spins of the order v / r, as a thermal aggregate has;
    a server's requests start without spin."""
    from libgran_gb300 import configs as K
    mat = K.Material()
    sizes = _sizes(case)
    x, v = K.seeded_aggregates(sizes, seed, mat.r, VMAX)
    om = np.random.default_rng(seed).uniform(-VMAX / mat.r, VMAX / mat.r, size=x.shape)
    if case["serve"]:
        om[:] = 0.0
    if case["wall"]:
        x = K.rest_on_wall(x, sizes, mat.r)
    return mat, sizes, x, v, om


def _r_verlet(case, mat):
    return 4.5 * mat.r if case["ham"] != "none" else 3.0 * mat.r


def _desc(case, mat, n):
    from libgran_gb300 import _abi as A
    from libgran_gb300 import configs as K
    model = {"contact": A.LG_BINARY_CONTACT, "sinter": A.LG_BINARY_SINTER, "breaking": A.LG_BINARY_BREAKING_SINTER}
    ham = {"none": A.LG_HAMAKER_NONE, "full": A.LG_HAMAKER_FULL, "limited": A.LG_HAMAKER_LIMITED}
    verlet = case["pairs"] == "verlet"
    return K.make_desc(
        n, model[case["model"]], ham[case["ham"]], contact=mat.contact(),
        sinter=None if case["model"] == "contact" else mat.sinter(),
        hamaker=None if case["ham"] == "none" else mat.hamaker(),
        pairs=A.LG_PAIRS_VERLET if verlet else A.LG_PAIRS_ALL, r_verlet=_r_verlet(case, mat) if verlet else 0.0,
        precision=A.LG_PRECISION_MIXED if case["precision"] == "mixed" else A.LG_PRECISION_FP64,
        n_facets=1 if case["wall"] else 0, facet_auto_move=1 if case["wall"] else 0,
        max_neighbors=96 if case["serve"] else 0)


def _wall_extent(mat, sizes):
    return 2.0 * mat.r * float(max(sizes))


def prepare(case, seed):
    from libgran_gb300 import configs as K
    from libgran_gb300.serving import Server
    from libgran_gb300.system import System
    mat, sizes, x, v, om = _inputs(case, seed)
    n = len(x)
    if case["serve"]:
        srv = Server(_desc(case, mat, 1), budget_bytes=8 * 10 ** 9, dt=mat.dt, rebuild_every=REBUILD)
        srv.set_slots([c for c in (128, 256, 512, 1024) for _ in range(6)])
        cut = np.concatenate([[0], np.cumsum(sizes)])
        reqs = [(x[a:b], v[a:b]) for a, b in zip(cut[:-1], cut[1:])]
        return dict(case=case, server=srv, requests=reqs)
    desc = _desc(case, mat, n)
    facets = [K.wall_facet(mat, _wall_extent(mat, sizes), V_WALL)] if case["wall"] else None
    neck = None
    if case["model"] == "breaking":
        # one strength per bond: the number of touching pairs, system by system
        neck = np.full(_count_bonds(x, sizes, mat), STRENGTH)
    sys = System(desc, x, v, om0=om, facets=facets, neck=neck, sizes=sizes if _batched(case) else None)
    # page-locked buffers that receive the state, as a driver that dumps regularly keeps
    out = tuple(torch.empty(n, 3, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
                for _ in range(4))
    return dict(case=case, system=sys, dt=mat.dt, out=out)


def run(state):
    case = state["case"]
    if case["serve"]:
        srv = state["server"]
        ids = [srv.submit(x, v, case["steps"]) for x, v in state["requests"]]
        while True:
            active, queued, _ = srv.tick()
            if active == 0 and queued == 0:
                break
        done = [srv.poll(q, want_x=True) for q in ids]
        for q in ids:
            srv.release(q)
        return {"x": np.concatenate([d["x"] for d in done]),
                "ke": np.array([d["obs"]["ke_total"] for d in done])}
    from libgran_gb300 import _abi as A
    sys = state["system"]
    every = REBUILD if case["pairs"] == "verlet" else 0
    for _ in range(case["calls"]):
        sys.step(state["dt"], case["steps"], every)
    x, v, th, om = sys.get_state(out=state["out"])
    got = {"x": x, "v": v, "theta": th, "omega": om}
    if case["obs"]:
        o = sys.observables(A.LG_OBS_STATE)
        got["obs"] = np.array([o["ke_translational"], o["ke_rotational"], o["linear_momentum"],
                               o["angular_momentum"], o["radius_of_gyration"]])
    return got


# ------------------------------------------------------------------------------------------------
# Work of one interval
# ------------------------------------------------------------------------------------------------
def work(case):
    """Per particle and step: state in and out (x, v, omega read; a, alpha, v, omega written: 168 B),
    the row's partner indices (4 B each) and the springs of its touching or bonded pairs (9 values
    read and written, 144 B each); once per interval the state that the caller reads (96 B). An
    aggregate of this kind holds about 23 partners within 4.5 r, 17 of them within the Hamaker cutoff
    of 4 r, and 1.9 touching. Operations: 60 per Hamaker pair, 400 per contact, 60 per particle; each
    unordered pair once."""
    if not _batched(case):
        n = float(case["n"])
    elif case["n"]:
        z = math.log(case["hi"] / case["n"]) / 2.326347874040841
        n = case["count"] * case["n"] * math.exp(0.5 * z * z)
    else:
        n = case["count"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    steps = case["steps"] * case["calls"]
    every = case["pairs"] == "all"
    ham = {"none": 0.0, "full": max(n - 1.0, 0.0) if every else 23.0, "limited": min(17.0, n - 1.0)}[case["ham"]]
    row = 0.0 if every else (23.0 if case["ham"] != "none" else 8.0)
    live = 1.9
    return {"bytes": n * (steps * (168.0 + 4.0 * row + 144.0 * live) + 96.0),
            "flops": n * steps * (60.0 * ham / 2 + 400.0 * live / 2 + 60.0)}


# ------------------------------------------------------------------------------------------------
# Plain FP64 evaluation
# ------------------------------------------------------------------------------------------------
def _near_pairs(x, sizes, reach):
    """Ordered pairs (i, j) of one system within `reach` of each other, i ascending (numpy)."""
    n = len(x)
    sysid = np.repeat(np.arange(len(sizes)), sizes)
    off = np.concatenate([[0], np.cumsum(sizes)])[:-1]
    lo = np.minimum.reduceat(x, off, axis=0)[sysid]
    cell = np.floor((x - lo) / reach).astype(np.int64) + 1
    dim = cell.max(0) + 2
    key = ((sysid * dim[2] + cell[:, 2]) * dim[1] + cell[:, 1]) * dim[0] + cell[:, 0]
    order = np.argsort(key, kind="stable")
    skey = key[order]
    out_i, out_j = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            shift = (dz * dim[1] + dy) * dim[0]  # the three cells along x are consecutive keys
            b = np.searchsorted(skey, key + shift - 1, side="left")
            e = np.searchsorted(skey, key + shift + 1, side="right")
            for at in range(0, n, 65536):
                bb, cnt = b[at:at + 65536], (e - b)[at:at + 65536]
                i = np.repeat(np.arange(at, at + len(cnt)), cnt)
                j = order[np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(bb, cnt)]
                d = x[i] - x[j]
                ok = (i != j) & ((d * d).sum(1) <= reach * reach)
                out_i.append(i[ok])
                out_j.append(j[ok])
    i, j = np.concatenate(out_i), np.concatenate(out_j)
    o = np.lexsort((j, i))
    return i[o], j[o]


def _bond_gap(x, i, j, r):
    d = x[i] - x[j]
    return np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) - 2.0 * r


def _count_bonds(x, sizes, mat):
    i, j = _near_pairs(x, sizes, 2.0 * mat.r + 2.0 * mat.d_crit)
    return int((np.abs(_bond_gap(x, i, j, mat.r)[i < j]) < mat.d_crit).sum())


def _bonded(x, i, j, mat, cycle_free):
    """Bonds among the ordered pairs: touching pairs, in (i, j) order, without closing a cycle for
    the plain sintered bond."""
    touch = np.abs(_bond_gap(x, i, j, mat.r)) < mat.d_crit
    if not cycle_free:
        return touch
    parent = list(range(len(x)))

    def root(a):
        while parent[a] != a:
            parent[a] = parent[parent[a]]
            a = parent[a]
        return a

    kept = set()
    for a, b in zip(i[touch & (i < j)].tolist(), j[touch & (i < j)].tolist()):
        ra, rb = root(a), root(b)
        if ra != rb:
            parent[rb] = ra
            kept.add((a, b))
    got = touch.copy()
    at = np.nonzero(touch)[0]
    got[at] = [(min(a, b), max(a, b)) in kept for a, b in zip(i[at].tolist(), j[at].tolist())]
    return got


def _dot(a, b):
    return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]


def _norm(a):
    return torch.sqrt(_dot(a, a))


def _unit(a):
    z = _norm(a)
    return torch.where((z > 0)[:, None], a / torch.where(z > 0, z, torch.ones_like(z))[:, None], a)


def _cross(a, b):
    return torch.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                        a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], 1)


def _shear(xi, n, k, g, fn, mu, phi, rel, dt, coulomb):
    """Shear spring (tangential, rolling or torsion): rotated onto the tangent plane at its length,
    stretched by the slip; with Coulomb friction capped. Returns (force, new spring)."""
    new = xi - _dot(xi, n)[:, None] * n
    xi = torch.where((_norm(new) > 0)[:, None], _norm(xi)[:, None] * _unit(new), new)
    f0 = -k * xi - g * rel
    stick = xi + dt * rel
    if not coulomb:
        return f0, stick
    f0n = _norm(f0)
    t = torch.where((f0n > 0)[:, None], _unit(f0), torch.zeros_like(f0))
    fs, fd = mu * fn, mu * phi * fn
    held = f0n <= fs
    slide = -1.0 / k * (fd[:, None] * t + g * rel)
    cap = torch.minimum(f0n, torch.where(held, fs, fd))
    return cap[:, None] * t, torch.where(held[:, None], stick, slide)


class _Plain:
    """The force laws and the velocity-Verlet loop on torch FP64 tensors, one entry per ordered pair."""

    def __init__(self, case, mat, sizes, x, v, om):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        self.case, self.mat, self.c = case, mat, mat.contact()
        n = len(x)
        every = case["pairs"] == "all" and case["ham"] == "full"
        if every:
            i = np.repeat(np.arange(n), n - 1)
            j = np.tile(np.arange(n - 1), n)
            j = j + (j >= i)
        else:  # pairs beyond the reach of every force add nothing
            reach = 1.001 * mat.r_cut if case["ham"] == "limited" else 2.2 * mat.r
            i, j = _near_pairs(x, sizes, reach)
        bonded = np.zeros(len(i), dtype=bool)
        if case["model"] != "contact":
            bonded = _bonded(x, i, j, mat, case["model"] == "sinter")
        self.i, self.j = t(i), t(j)
        near = bonded | (((x[i] - x[j]) ** 2).sum(1) < (2.2 * mat.r) ** 2)
        self.near = t(np.nonzero(near)[0])  # pairs that can touch during the interval
        self.bonded = t(bonded[near])
        self.xi = [torch.zeros(int(near.sum()), 3, dtype=torch.float64, device=self.dev) for _ in range(3)]
        self.x, self.v, self.om = t(x.copy()), t(v.copy()), t(om.copy())
        self.th = torch.zeros(n, 3, dtype=torch.float64, device=self.dev)
        if case["wall"]:
            L = 20.0 * _wall_extent(mat, sizes)
            self.vert = [torch.tensor(p, dtype=torch.float64) for p in
                         ((-L, -L, 0.0), (-L, 3 * L, 0.0), (3 * L, -L, 0.0))]
            first = [p.reshape(1, 3).to(self.dev) for p in self.vert]
            self.cross0 = _cross(first[1] - first[0], first[2] - first[0])
            self.sxi = [torch.zeros(n, 3, dtype=torch.float64, device=self.dev) for _ in range(3)]
        self.a, self.al = self.forces()

    def contact_like(self, n, overlap, dv, wi, wj, xi, bonded):
        """Accelerations of touching or bonded pairs (the sintered bond shares the contact's constants
        and has no Coulomb cap) and their new springs."""
        c = self.c
        rp = c.r_part - overlap / 2.0
        fn = c.k * overlap + c.gamma_n * -_dot(dv, n)
        nwi, nwj = _cross(n, wi), _cross(n, wj)
        vij = dv + rp[:, None] * nwi + rp[:, None] * nwj
        vt = vij - _dot(vij, n)[:, None] * n
        vr = -rp[:, None] * (nwi - nwj)
        vo = (c.r_part * (_dot(n, wi) - _dot(n, wj)))[:, None] * n
        out = []
        for s, (k, g, mu, phi, rel) in zip(xi, ((c.k_t, c.gamma_t, c.mu_s, c.phi_d, vt),
                                                (c.k_r, c.gamma_r, c.mu_r, c.phi_r, vr),
                                                (c.k_o, c.gamma_o, c.mu_o, c.phi_o, vo))):
            f, new = _shear(s, n, k, g, fn, mu, phi, rel, c.dt, True)
            fb, newb = _shear(s, n, k, g, fn, mu, phi, rel, c.dt, False)
            out.append((torch.where(bonded[:, None], fb, f), torch.where(bonded[:, None], newb, new)))
        (ft, s0), (fr, s1), (fo, s2) = out
        tau = -(rp[:, None] * _cross(n, ft)) + c.r_part * _cross(n, fr) + c.r_part * fo
        return fn[:, None] * n + ft, tau, [s0, s1, s2]

    def forces(self):
        m, c, n = self.mat, self.c, len(self.x)
        a, al = torch.zeros_like(self.x), torch.zeros_like(self.x)
        i, j = self.i[self.near], self.j[self.near]
        dx = self.x[i] - self.x[j]
        nn = _unit(dx)
        overlap = 2.0 * c.r_part - _dot(dx, nn)
        on = self.bonded | ~(overlap <= 0)
        f, tau, xi = self.contact_like(nn, overlap, self.v[i] - self.v[j], self.om[i], self.om[j], self.xi, self.bonded)
        self.xi = [torch.where(on[:, None], s, torch.zeros_like(s)) for s in xi]
        keep = on[:, None].to(torch.float64)
        a.index_add_(0, i, keep * f / c.mass)
        al.index_add_(0, i, keep * tau / c.inertia)
        if self.case["model"] == "breaking":
            broken = self.bonded & (_norm(f) > STRENGTH)
            self.bonded = self.bonded & ~broken
            self.xi = [torch.where(broken[:, None], torch.zeros_like(s), s) for s in self.xi]
        if self.case["ham"] != "none":
            for at in range(0, len(self.i), 1 << 22):
                i, j = self.i[at:at + (1 << 22)], self.j[at:at + (1 << 22)]
                r = self.x[j] - self.x[i]
                d = _norm(r)
                h = torch.clamp(d - 2.0 * m.r, min=m.h0)
                q, w, p = 4.0 * m.r + h, 2.0 * m.r + h, 4.0 * m.r + 2.0 * h
                br = p / q / h - 2.0 / w - 4.0 * m.r ** 2 / (w * w * w) - 2.0 * m.r ** 2 * p / (q * q) / (h * h)
                s = -m.A / 6.0 * br
                if self.case["ham"] == "limited":
                    s = torch.where(d > m.r_cut, torch.zeros_like(s), s)
                a.index_add_(0, i, s[:, None] * (r / d[:, None]) / m.m)
        if self.case["wall"]:
            fa, fal = self.wall()
            a, al = a + fa, al + fal
        return a, al

    def nearest_on_wall(self):
        """libgran's nearest point of the triangle: the projection onto its plane where the three
        partial areas add up to no more than the triangle's (to the last bit), else the nearest point
        of an edge."""
        p = self.x
        vert = [q.to(self.dev).reshape(1, 3) for q in self.vert]
        N = _unit(self.cross0)
        rows = lambda q: q.expand_as(p)  # noqa: E731
        foot = (p - _dot(p, rows(N))[:, None] * N) + _dot(vert[0], N)[:, None] * N
        to = [rows(q) - foot for q in vert]
        area = 0.5 * _norm(_cross(to[0], to[1])) + 0.5 * _norm(_cross(to[1], to[2])) + 0.5 * _norm(_cross(to[2], to[0]))
        edge = []
        for k in range(3):
            a, b = vert[k], vert[(k + 1) % 3]
            along = _unit(b - a)
            at = _dot(p - a, rows(along))[:, None]
            q = torch.where(at > _norm(b - a)[:, None], rows(b), a + at * along)
            edge.append(torch.where(at < 0, rows(a), q))
        d = [_dot(p - q, p - q)[:, None] for q in edge]
        first = (d[0] < d[1]) & (d[0] < d[2])
        second = ~(d[0] < d[1]) & (d[1] < d[2])
        out = torch.where(first, edge[0], torch.where(second, edge[1], edge[2]))
        return torch.where((area > 0.5 * _norm(self.cross0))[:, None], out, foot)

    def wall(self):
        c, m = self.c, self.mat
        foot = self.nearest_on_wall()
        p = self.x
        dx = p - foot
        n = _unit(dx)
        overlap = c.r_part - _dot(dx, n)
        vf = torch.tensor([[0.0, 0.0, V_WALL]], dtype=torch.float64, device=self.dev)
        rp = c.r_part - overlap
        fn = c.k * overlap + c.gamma_n * -_dot(self.v - vf, n)
        nwi = _cross(n, self.om)
        vij = self.v - vf + rp[:, None] * nwi
        vt = vij - _dot(vij, n)[:, None] * n
        vr = -rp[:, None] * nwi
        vo = (c.r_part * _dot(n, self.om))[:, None] * n
        ft, s0 = _shear(self.sxi[0], n, c.k_t, c.gamma_t, fn, c.mu_s, c.phi_d, vt, c.dt, True)
        fr, s1 = _shear(self.sxi[1], n, c.k_r, c.gamma_r, fn, c.mu_r, c.phi_r, vr, c.dt, True)
        fo, s2 = _shear(self.sxi[2], n, c.k_o, c.gamma_o, fn, c.mu_o, c.phi_o, vo, c.dt, True)
        on = (~(overlap <= 0))[:, None].to(torch.float64)
        self.sxi = [on * s for s in (s0, s1, s2)]
        fa = on * (fn[:, None] * n + ft) / c.mass
        fal = on * (-(rp[:, None] * _cross(n, ft)) + c.r_part * _cross(n, fr) + c.r_part * fo) / c.inertia
        r = foot - p
        h = torch.clamp(_norm(r) - m.r, min=m.h0)
        s = 2.0 * m.A / 3.0 * (m.r ** 3 / (h * h) / ((h + 2.0 * m.r) * (h + 2.0 * m.r)))
        return fa + s[:, None] * _unit(r) / m.m, fal

    def step(self, dt):
        h = dt / 2.0
        self.v, self.om = self.v + h * self.a, self.om + h * self.al
        self.x, self.th = self.x + dt * self.v, self.th + dt * self.om
        self.a, self.al = self.forces()
        self.v, self.om = self.v + h * self.a, self.om + h * self.al
        if self.case["wall"]:
            self.vert = [p + torch.tensor([0.0, 0.0, V_WALL * dt], dtype=torch.float64) for p in self.vert]


def exact(case, seed):
    mat, sizes, x, v, om = _inputs(case, seed)
    if not torch.cuda.is_available() and len(x) * case["steps"] * case["calls"] > 400000:
        return None  # minutes on a CPU
    s = _Plain(case, mat, sizes, x, v, om)
    for _ in range(case["steps"] * case["calls"]):
        s.step(mat.dt)
    if case["serve"]:
        e = 0.5 * mat.m * (s.v * s.v).sum(1) + 0.5 * mat.I * (s.om * s.om).sum(1)
        sysid = torch.as_tensor(np.repeat(np.arange(len(sizes)), sizes), device=s.dev)
        ke = torch.zeros(len(sizes), dtype=torch.float64, device=s.dev).index_add_(0, sysid, e)
        return {"x": s.x.cpu().numpy(), "ke": ke.cpu().numpy()}
    got = {k: a.cpu().numpy() for k, a in (("x", s.x), ("v", s.v), ("theta", s.th), ("omega", s.om))}
    if case["obs"]:
        xx, vv, ww = got["x"], got["v"], got["omega"]
        com = xx.mean(0)
        got["obs"] = np.array([
            0.5 * mat.m * (vv * vv).sum(), 0.5 * mat.I * (ww * ww).sum(), np.linalg.norm(mat.m * vv.sum(0)),
            np.linalg.norm((mat.I * ww + mat.m * np.cross(xx, vv)).sum(0)),
            math.sqrt(((xx - com) ** 2).sum(1).mean())])
    return got
