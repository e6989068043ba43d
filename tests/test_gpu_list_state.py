"""The Verlet list's two buffers (the current list, and the idle one that holds scratch between builds) over every
way that a handle is stepped. The same operations run in each, so the tolerance is zero."""
import os
import subprocess
import time

import numpy as np
import pytest

from libgran_gb300 import _abi as A
from libgran_gb300 import configs as K
from libgran_gb300.serving import Server
from libgran_gb300.system import System, generate_aggregate, generate_velocities

import helpers as H

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRECISIONS = pytest.mark.parametrize("precision", [A.LG_PRECISION_FP64, A.LG_PRECISION_MIXED], ids=["fp64", "mixed"])


def _system(n, precision, pairs=A.LG_PAIRS_VERLET, bm=A.LG_BINARY_CONTACT):
    mat = K.Material()
    x0 = generate_aggregate(21, n, mat.r)
    v0 = generate_velocities(21, n, 0.1) - 2e7 * (x0 - x0.mean(0))
    d = K.make_desc(n, bm, A.LG_HAMAKER_LIMITED, contact=mat.contact(), sinter=mat.sinter(), hamaker=mat.hamaker(),
                    pairs=pairs, r_verlet=4.5 * mat.r if pairs == A.LG_PAIRS_VERLET else 0.0, precision=precision,
                    max_neighbors=96)
    return System(d, x0, v0)


@PRECISIONS
@pytest.mark.parametrize("pairs,n", [(A.LG_PAIRS_VERLET, 300), (A.LG_PAIRS_VERLET, 900), (A.LG_PAIRS_ALL, 70)],
                         ids=["verlet-300", "verlet-900", "all-70"])
def test_steps_without_rebuilds_between_steps_with_them(pairs, n, precision):
    """A run without rebuilds is captured sixteen steps at a time, and so is one that rebuilds every sixteen: the
    two graphs differ in what they do to the lists."""
    dt = K.Material().dt
    schedule = [(48, 0), (48, 16), (48, 0), (1, 0), (47, 16), (32, 16), (5, 0), (32, 0)]
    runs = []
    for graphs in (True, False):
        s = _system(n, precision, pairs)
        s.set_graphs(graphs)
        out = []
        for nst, rb in schedule:
            s.step(dt, nst, rb)
            out += [s.get(f) for f in H.FIELDS]
        assert s.device_errors() == 0
        runs.append(out)
        s.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b), H.rel_err(a, b)


@PRECISIONS
@pytest.mark.parametrize("kind", ["batch-on-a-wall", "all-pairs-bonds"])
def test_every_creation_sees_its_uploads(kind, precision):
    """The construction's force evaluation runs on the handle's own stream, after the copies of the systems' offsets,
    the facets' vertices and the pair flags."""
    mat = K.Material()
    wall = kind == "batch-on-a-wall"
    sizes = np.array([40, 1, 300, 7] if wall else [120])
    x0 = np.concatenate([generate_aggregate(31 + q, n, mat.r) for q, n in enumerate(sizes)])
    if wall:
        x0 = K.rest_on_wall(x0, sizes, mat.r)
    d = K.make_desc(len(x0), A.LG_BINARY_SINTER, A.LG_HAMAKER_LIMITED, contact=mat.contact(), sinter=mat.sinter(),
                    hamaker=mat.hamaker(), pairs=A.LG_PAIRS_VERLET if wall else A.LG_PAIRS_ALL,
                    r_verlet=4.5 * mat.r if wall else 0.0, precision=precision, max_neighbors=96, n_facets=1 if wall else 0)
    first = None
    for _ in range(20):
        s = System(d, x0, sizes=sizes if wall else None, facets=[K.wall_facet(mat, 200 * mat.r)] if wall else None)
        a = s.get(A.LG_FIELD_A)
        first = a if first is None else first
        assert np.array_equal(a, first)
        s.close()


def _cpp(tmp_path, name, *args):
    """Builds tests/cpp/<name>.cpp against the engine's library and its internal header, and runs it."""
    so, cuda = A.lib()._name, os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = tmp_path / name
    subprocess.run([os.path.join(cuda, "bin", "nvcc"), "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "libgran_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", name + ".cpp"), so, "-Xlinker", "-rpath=" + os.path.dirname(so),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)] + list(args), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[:2000] + r.stderr
    return r.stdout.split()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_slot_emptied_between_builds_owns_no_pairs(tmp_path, precision):
    b0, b1, a0, a1, same, errs = (int(v) for v in _cpp(tmp_path, "arena_owners", precision))
    assert b0 > 0 and b0 == b1 and a0 == 0 and a1 == b1
    assert same and errs == 0


@PRECISIONS
def test_served_budgets_that_end_between_builds(precision):
    """Requests retire between two list builds; the others, and later occupants of their slots, end as lone runs do."""
    mat = K.Material()
    d = K.make_desc(1, A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, contact=mat.contact(), hamaker=mat.hamaker(),
                    pairs=A.LG_PAIRS_VERLET, r_verlet=4.5 * mat.r, precision=precision, max_neighbors=96)
    srv = Server(d, budget_bytes=4 * 10 ** 9, dt=mat.dt, rebuild_every=20)
    srv.set_slots([128, 256, 256])
    jobs = [(100, 7), (200, 55), (250, 40), (90, 33), (180, 61), (256, 13)]
    states = [(generate_aggregate(40 + q, n, mat.r), generate_velocities(40 + q, n, 0.1)) for q, (n, _) in enumerate(jobs)]
    ids = [srv.submit(x, v, steps) for (x, v), (_, steps) in zip(states, jobs)]
    for _ in range(200):
        active, queued, _ = srv.tick()
        if active == 0 and queued == 0:
            break
    for (n, steps), (x, v), q in zip(jobs, states, ids):
        got = srv.poll(q, want_x=True)
        d.n_part = n
        d.force_kernel = A.LG_FORCE_KERNEL_COMPACT
        s = System(d, x, v)
        s.step(mat.dt, steps, 20)
        want = s.get(A.LG_FIELD_X)
        s.close()
        if precision == A.LG_PRECISION_FP64:
            assert np.array_equal(got["x"], want), (n, steps)
        else:  # a run's float-float state is rounded to FP64 where the run ends, at another step than the lone run's
            assert H.rel_err(got["x"] - x, want - x) <= 1e-5, (n, steps)


@PRECISIONS
def test_lists_of_systems_shared_by_several_blocks(precision):
    """A batch's systems take blocks by their sizes: around one block's share, and far beyond it."""
    sizes = np.array([255, 256, 257, 1, 513, 9000])
    mat = K.Material()
    xs = [generate_aggregate(60 + q, n, mat.r) for q, n in enumerate(sizes)]

    def system(x, batch):
        d = K.make_desc(len(x), A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, contact=mat.contact(), hamaker=mat.hamaker(),
                        pairs=A.LG_PAIRS_VERLET, r_verlet=4.5 * mat.r, precision=precision, max_neighbors=96,
                        force_kernel=A.LG_FORCE_KERNEL_COMPACT)
        s = System(d, x, generate_velocities(3, len(x), 0.1) * 0.0, sizes=sizes if batch else None)
        for _ in range(3):
            s.update_neighbor_list()
        s.step(mat.dt, 1, 0)
        out, st = s.get(A.LG_FIELD_A), s.pair_stats()
        assert s.device_errors() == 0
        s.close()
        return out, st["mean_row_length"] * len(x)

    got, rows = system(np.concatenate(xs), True)
    cut = np.concatenate([[0], np.cumsum(sizes)])
    alone = [system(x, False) for x in xs]
    assert rows == pytest.approx(sum(r for _, r in alone), rel=1e-12)
    for q, (want, _) in enumerate(alone):
        if precision == A.LG_PRECISION_FP64:
            assert np.array_equal(got[cut[q]:cut[q + 1]], want), q
        elif np.abs(want).max() > 0:  # sums are grouped by the launch's slicing, a function of the total size
            assert H.rel_err(got[cut[q]:cut[q + 1]], want) <= 1e-6, q


def test_a_large_system_of_a_batch_builds_its_list_as_fast_as_alone():
    """The build's passes are shared out by particles: a batch that is nearly all one system takes about as long as
    that system (1.1 times, measured; with one block per system it took 2.5 times as long)."""
    mat = K.Material()
    n = 100000
    x = np.concatenate([generate_aggregate(5, n, mat.r), generate_aggregate(6, 500, mat.r)])

    def build_time(x, sizes):
        d = K.make_desc(len(x), A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, contact=mat.contact(), hamaker=mat.hamaker(),
                        pairs=A.LG_PAIRS_VERLET, r_verlet=4.5 * mat.r, precision=A.LG_PRECISION_MIXED)
        s = System(d, x, sizes=sizes)
        best = np.inf
        for _ in range(6):
            s.device_errors()
            t0 = time.perf_counter()
            for _ in range(20):
                s.update_neighbor_list()
            s.device_errors()
            best = min(best, time.perf_counter() - t0)
        s.close()
        return best

    assert build_time(x, [n, 500]) <= 1.6 * build_time(x[:n], None)


@pytest.mark.parametrize("bm", [A.LG_BINARY_CONTACT, A.LG_BINARY_SINTER], ids=["contact", "sinter"])
@pytest.mark.parametrize("n", [511, 512, 4096, 4097, 23999, 24001, 32769])
def test_contacts_evaluated_once_per_pair_equal_rows(n, bm):
    """Candidates near contact are evaluated once per pair, in blocks of 32, 64 or 128 rows; the persistent kernel
    evaluates each order by itself."""
    mat = K.Material()
    x0 = generate_aggregate(70, n, mat.r)
    v0 = generate_velocities(70, n, 0.1) - 2e7 * (x0 - x0.mean(0))
    runs = []
    for kernel in (A.LG_FORCE_KERNEL_PERSISTENT, A.LG_FORCE_KERNEL_COMPACT):
        for rv in (4.1, 4.5):
            d = K.make_desc(n, bm, A.LG_HAMAKER_LIMITED, contact=mat.contact(), sinter=mat.sinter(), hamaker=mat.hamaker(),
                            pairs=A.LG_PAIRS_VERLET, r_verlet=rv * mat.r, precision=A.LG_PRECISION_MIXED, max_neighbors=96,
                            force_kernel=kernel)
            s = System(d, x0, v0)
            s.step(mat.dt, 1, 20)
            s.step(mat.dt, 39, 20)
            assert s.device_errors() == 0
            runs.append([s.get(f) for f in H.FIELDS])
            s.close()
    for a, b in ((runs[0], runs[2]), (runs[1], runs[3])):
        for u, v in zip(a, b):
            assert np.array_equal(u, v), H.rel_err(u, v)


def test_staged_handles_take_what_they_need(tmp_path):
    """One chunk from the pool that holds every buffer of the handle (a monomer's bonds: 8 reckoned, 1 to 7 used) and
    nothing else of note; the server charges it and a fixed 4 MiB."""
    rows = np.array([int(v) for v in _cpp(tmp_path, "staged_bytes")]).reshape(-1, 7)
    assert len(rows) == 24
    for precision, model, n, chunk, used, chunks, charged in rows:
        assert chunks == 1, (precision, model, n)
        assert chunk - used <= 64 * 1024 + 0.05 * chunk, (precision, model, n, chunk, used)
        assert chunk <= charged <= chunk + 2 ** 22


@pytest.mark.parametrize("n,wall", [(2499, False), (2501, False), (8500, False), (8501, False), (16383, False),
                                    (16385, False), (8999, True), (9001, True)], ids=str)
def test_fp64_pair_kernels_equal_rows_at_their_launch_lines(n, wall):
    """The row kernel at one thread per row adds each row in index order, and so do the pair kernels, whatever their block
    shapes: the same bits."""
    mat = K.Material()
    x0 = generate_aggregate(90, n, mat.r)
    v0 = generate_velocities(90, n, 0.1) - 2e7 * (x0 - x0.mean(0))
    if wall:
        x0 = K.rest_on_wall(x0, np.array([n]), mat.r)
    runs = []
    for kernel in (A.LG_FORCE_KERNEL_ROWGROUP, A.LG_FORCE_KERNEL_AUTO):
        d = K.make_desc(n, A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, contact=mat.contact(), hamaker=mat.hamaker(),
                        pairs=A.LG_PAIRS_VERLET, r_verlet=4.5 * mat.r, max_neighbors=96, force_kernel=kernel,
                        threads_per_row=1 if kernel == A.LG_FORCE_KERNEL_ROWGROUP else 0, n_facets=1 if wall else 0,
                        facet_auto_move=1 if wall else 0)
        s = System(d, x0, v0, facets=[K.wall_facet(mat, 200 * mat.r, 1.0)] if wall else None)
        s.step(mat.dt, 1, 5)
        s.step(mat.dt, 11, 5)
        assert s.device_errors() == 0
        runs.append([s.get(f) for f in H.FIELDS])
        s.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b), H.rel_err(a, b)


def test_tuned_handles_hold_no_graph_of_another_shape(tmp_path):
    held, eager, replayed = (int(v) for v in _cpp(tmp_path, "tuned_graphs"))
    assert held == 0 and eager == replayed


@PRECISIONS
def test_a_server_emptied_between_boundaries_goes_on_admitting(precision):
    """Every request of a wave ends between two list builds, with others queued behind it, and a later wave finds the
    server idle there: each ends as its lone run does (FP64: the same bits)."""
    mat = K.Material()
    d = K.make_desc(1, A.LG_BINARY_SINTER, A.LG_HAMAKER_LIMITED, contact=mat.contact(), sinter=mat.sinter(),
                    hamaker=mat.hamaker(), pairs=A.LG_PAIRS_VERLET, r_verlet=4.5 * mat.r, precision=precision,
                    max_neighbors=96)
    srv = Server(d, budget_bytes=4 * 10 ** 9, dt=mat.dt, rebuild_every=20)
    srv.set_slots([128])
    for wave in range(2):
        jobs = [(60 + 20 * q, 7 + 19 * q) for q in range(3)]
        states = [(generate_aggregate(90 + q, n, mat.r), generate_velocities(90 + wave, n, 0.1)) for q, (n, _) in enumerate(jobs)]
        ids = [srv.submit(x, v, steps) for (x, v), (_, steps) in zip(states, jobs)]
        for _ in range(100):
            active, queued, _ = srv.tick()
            if active == 0 and queued == 0:
                break
        for (n, steps), (x, v), q in zip(jobs, states, ids):
            got = srv.poll(q, want_x=True)
            assert got["state"] == A.LG_REQ_DONE, (wave, n)
            d.n_part = n
            s = System(d, x, v)
            s.step(mat.dt, steps, 20)
            want = s.get(A.LG_FIELD_X)
            s.close()
            if precision == A.LG_PRECISION_FP64:
                assert np.array_equal(got["x"], want), (wave, n)
            else:
                assert H.rel_err(got["x"] - x, want - x) <= 1e-5, (wave, n)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("shape", ["chain", "plane", "rod"])
def test_lists_of_stretched_systems_hold_every_pair(shape, axis):
    """Long lines of cells along x are laid along the thinnest axis. In FP64 the forces over the list equal the forces over
    all pairs, whose partners out of range add zeros: the same bits."""
    mat = K.Material()
    n, r = 6000, mat.r
    q = np.arange(n)
    rng = np.random.default_rng(4)
    if shape == "chain":
        x0 = np.stack([1.999 * r * q, 0 * q, 0 * q], 1)
    elif shape == "plane":
        x0 = np.stack([rng.random(n) * 1500 * r, rng.random(n) * 60 * r, 0 * q], 1)
    else:
        x0 = np.stack([1.999 * r * (q // 4), 2.1 * r * (q % 2), 2.2 * r * ((q // 2) % 2)], 1) + 0.1 * r * rng.random((n, 3))
    x0 = np.ascontiguousarray(np.roll(x0, axis, 1))
    acc = []
    for pairs in (A.LG_PAIRS_ALL, A.LG_PAIRS_VERLET):
        d = K.make_desc(n, A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, contact=mat.contact(), hamaker=mat.hamaker(), pairs=pairs,
                        r_verlet=4.5 * r if pairs == A.LG_PAIRS_VERLET else 0.0, max_neighbors=200 if pairs == A.LG_PAIRS_VERLET else 0)
        s = System(d, x0, generate_velocities(6, n, 0.1))
        if pairs == A.LG_PAIRS_VERLET:
            s.update_neighbor_list()
        s.step(mat.dt, 3, 2)
        assert s.device_errors() == 0
        acc.append([s.get(f) for f in H.FIELDS])
        s.close()
    for a, b in zip(*acc):
        assert np.array_equal(a, b), H.rel_err(a, b)


def test_a_chain_builds_its_list_as_fast_along_x_as_along_z():
    """(0.9 to 1.1 times, measured; 3.9 times when one warp walked the line of cells that a chain along x fills.)"""
    mat = K.Material()
    n = 20000
    best = []
    for axis in (0, 2):
        x0 = np.zeros((n, 3))
        x0[:, axis] = 2.0 * mat.r * np.arange(n)
        d = K.make_desc(n, A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, contact=mat.contact(), hamaker=mat.hamaker(),
                        pairs=A.LG_PAIRS_VERLET, r_verlet=4.5 * mat.r)
        s = System(d, x0)
        times = []
        for _ in range(6):
            s.device_errors()
            t0 = time.perf_counter()
            for _ in range(20):
                s.update_neighbor_list()
            s.device_errors()
            times.append(time.perf_counter() - t0)
        best.append(min(times))
        s.close()
    assert best[0] <= 2.0 * best[1]
