"""Kernels that evaluate each unordered pair once and hand the result to both rows, the list build and the
unary terms beside the pair kernels, at the sizes where their launch shapes change and on the rows that are
not symmetric. FP64 is compared with the row kernel at one thread per row (each row alone, in index order);
the mixed contacts with the persistent kernel (each order of a pair by itself). Both are the same arithmetic
in the same order of summation, so the tolerance is zero."""
import numpy as np
import pytest

from libgran_gb300 import _abi as A
from libgran_gb300 import configs as K
from libgran_gb300.system import System, generate_aggregate, generate_velocities

import helpers as H

pytestmark = pytest.mark.gpu


def _desc(n, bm, hm, pairs, kernel, precision=A.LG_PRECISION_FP64, **kw):
    mat = K.Material()
    d = K.make_desc(n, bm, hm, contact=mat.contact(), sinter=mat.sinter(), hamaker=mat.hamaker(), pairs=pairs,
                    r_verlet=4.5 * mat.r if pairs == A.LG_PAIRS_VERLET else 0.0, precision=precision,
                    force_kernel=kernel, **kw)
    d.threads_per_row = 1 if kernel == A.LG_FORCE_KERNEL_ROWGROUP else 0
    return mat, d


def _state(n, seed, squeeze=2e7, shift=0.0):
    mat = K.Material()
    x0 = generate_aggregate(seed, n, mat.r)
    return x0 + shift * mat.r, generate_velocities(seed, n, 0.1) - squeeze * (x0 - x0.mean(0))


def _run(d, x0, v0, schedule, neck=None, sizes=None, facets=None, graphs=True, errors=0):
    s = System(d, x0, v0, neck=neck, sizes=sizes, facets=facets)
    s.set_graphs(graphs)
    out = [s.get(A.LG_FIELD_A)]
    for nst, rb in schedule:
        s.step(K.Material().dt, nst, rb)
        out += [s.get(f) for f in H.FIELDS]
    assert s.device_errors() == errors
    s.close()
    return out


def _same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x, y), H.rel_err(x, y)


MODELS = [(A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED), (A.LG_BINARY_SINTER, A.LG_HAMAKER_FULL),
          (A.LG_BINARY_BREAKING_SINTER, A.LG_HAMAKER_LIMITED), (A.LG_BINARY_NONE, A.LG_HAMAKER_LIMITED),
          (A.LG_BINARY_CONTACT, A.LG_HAMAKER_NONE)]
MODEL_IDS = ["contact", "sinter", "breaking", "hamaker", "contact-only"]


@pytest.mark.parametrize("bm,hm", MODELS, ids=MODEL_IDS)
@pytest.mark.parametrize("pairs,n", [(A.LG_PAIRS_ALL, n) for n in (1, 2, 3, 33, 394, 395, 727, 1025)] +
                         [(A.LG_PAIRS_VERLET, n) for n in (1, 2, 11, 2499, 2501, 5001, 6000, 6001, 16383, 16385)],
                         ids=lambda v: str(v))
def test_fp64_pairs_equal_rows(pairs, n, bm, hm):
    x0, v0 = _state(n, 100 + n)
    rb = 5 if pairs == A.LG_PAIRS_VERLET else 0
    runs = []
    for kernel in (A.LG_FORCE_KERNEL_ROWGROUP, A.LG_FORCE_KERNEL_AUTO):
        mat, d = _desc(n, bm, hm, pairs, kernel, max_neighbors=96)
        neck = None
        if bm == A.LG_BINARY_BREAKING_SINTER:
            neck = np.full(len(System(d, x0, v0).bonds()) // 2, 2e-9)
        runs.append(_run(d, x0, v0, [(1, 0), (12, rb)], neck))
    _same(*runs)


@pytest.mark.parametrize("bm,hm", MODELS[:3], ids=MODEL_IDS[:3])
@pytest.mark.parametrize("cap", [2, 3, 7])
def test_fp64_pairs_equal_rows_where_lists_overflow(cap, bm, hm):
    """Truncated rows: a pair may be in one particle's row only. Which partners such a row keeps may differ
    between two builds, so both kernels step from one snapshot, on one list."""
    n = 3001
    x0, v0 = _state(n, 7)
    mat, d = _desc(n, bm, hm, A.LG_PAIRS_VERLET, A.LG_FORCE_KERNEL_AUTO, max_neighbors=cap)
    neck = None
    if bm == A.LG_BINARY_BREAKING_SINTER:
        neck = np.full(len(System(d, x0, v0).bonds()) // 2, 2e-9)
    s = System(d, x0, v0, neck=neck)
    s.step(mat.dt, 3, 0)
    assert s.device_errors() & A.LG_DEVERR_LIST_OVERFLOW
    s.snapshot()
    runs = []
    for kernel in (A.LG_FORCE_KERNEL_COMPACT, A.LG_FORCE_KERNEL_ROWGROUP):
        s.restore()
        s.set_force_kernel(kernel)
        if kernel == A.LG_FORCE_KERNEL_ROWGROUP:
            s.set_threads_per_row(1)
        s.step(mat.dt, 12, 0)
        runs.append([s.get(f) for f in H.FIELDS])
    _same(*runs)


def test_fp64_pairs_equal_rows_with_neck_strengths_by_reference_indexing():
    """The two orders of a pair then look up different strengths, and one may break before the other."""
    n = 2600
    x0, v0 = _state(n, 9)
    runs = []
    for kernel in (A.LG_FORCE_KERNEL_ROWGROUP, A.LG_FORCE_KERNEL_AUTO):
        mat, d = _desc(n, A.LG_BINARY_BREAKING_SINTER, A.LG_HAMAKER_LIMITED, A.LG_PAIRS_VERLET, kernel, max_neighbors=96)
        nb = len(System(d, x0, v0).bonds()) // 2  # unbreakable, so all that were detected
        d.neck_mode = A.LG_NECK_REFERENCE_INDEXING
        runs.append(_run(d, x0, v0, [(30, 10)], np.geomspace(5e-10, 5e-8, nb)))
    _same(*runs)


@pytest.mark.parametrize("precision,n", [(A.LG_PRECISION_FP64, 2600), (A.LG_PRECISION_MIXED, 8500)], ids=["fp64", "mixed"])
def test_restored_list_owns_its_pairs_again(precision, n):
    """A snapshot holds the list, not which row owns a pair: that is worked out again after a restore."""
    x0, v0 = _state(n, 13)
    mat, d = _desc(n, A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, A.LG_PAIRS_VERLET, A.LG_FORCE_KERNEL_AUTO, precision,
                   max_neighbors=96)
    s = System(d, x0, v0)
    s.step(mat.dt, 23, 20)
    s.snapshot()
    s.step(mat.dt, 9, 20)
    want = [s.get(f) for f in H.FIELDS]
    s.step(mat.dt, 60, 20)  # other lists since
    s.restore()
    s.step(mat.dt, 9, 20)
    _same([s.get(f) for f in H.FIELDS], want)


@pytest.mark.parametrize("bm,hm", [m for m in MODELS if m[0] != A.LG_BINARY_NONE],
                         ids=[i for i in MODEL_IDS if i != "hamaker"])
@pytest.mark.parametrize("n", [511, 513, 8191, 8193, 32767, 49153])
def test_mixed_pairs_equal_persistent_rows(n, bm, hm):
    x0, v0 = _state(n, 200 + n)
    runs = []
    for kernel in (A.LG_FORCE_KERNEL_PERSISTENT, A.LG_FORCE_KERNEL_COMPACT):
        mat, d = _desc(n, bm, hm, A.LG_PAIRS_VERLET, kernel, A.LG_PRECISION_MIXED, max_neighbors=96)
        neck = None
        if bm == A.LG_BINARY_BREAKING_SINTER:
            neck = np.full(len(System(d, x0, v0).bonds()) // 2, 2e-9)
        runs.append(_run(d, x0, v0, [(1, 20), (19, 20), (27, 20)], neck))
    _same(*runs)


@pytest.mark.parametrize("shift", [0.0, -3e3, 1e6], ids=lambda v: "%g" % v)
@pytest.mark.parametrize("precision", [A.LG_PRECISION_FP64, A.LG_PRECISION_MIXED], ids=["fp64", "mixed"])
def test_batch_lists_equal_lists_alone(precision, shift):
    """One grid per system: sizes from one particle, positions away from the origin, systems that overlap."""
    sizes = [1, 2, 3, 700, 31, 33, 1500, 1, 257, 64]
    xs, vs = zip(*[_state(n, 300 + q, shift=shift * (q % 3)) for q, n in enumerate(sizes)])
    mat, d = _desc(sum(sizes), A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, A.LG_PAIRS_VERLET, A.LG_FORCE_KERNEL_COMPACT,
                   precision, max_neighbors=96)
    got = _run(d, np.concatenate(xs), np.concatenate(vs), [(1, 5), (12, 5)], sizes=sizes)
    off = np.concatenate([[0], np.cumsum(sizes)])
    for q, n in enumerate(sizes):
        _, dq = _desc(n, A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, A.LG_PAIRS_VERLET, A.LG_FORCE_KERNEL_COMPACT, precision,
                      max_neighbors=96)
        want = _run(dq, xs[q], vs[q], [(1, 5), (12, 5)])
        if precision == A.LG_PRECISION_FP64:
            for a, b in zip(got, want):
                assert np.array_equal(a[off[q]:off[q + 1]], b), q
        elif np.abs(want[0]).max() > 0:  # sums are grouped by the launch's slicing, a function of the total size
            assert H.rel_err(got[0][off[q]:off[q + 1]], want[0]) <= 1e-6, q


@pytest.mark.parametrize("count", [1, 40], ids=["one", "grid-stride"])
def test_mixed_unary_terms_beside_the_pairs(count):
    """Facet and body terms from their own stream: the same eagerly, graph-replayed and in a batch larger than
    the unary kernel's grid (152 x 8 blocks of 64), and within 1e-6 of the FP64 path."""
    n = 2000
    mat = K.Material()
    x0, v0 = _state(n, 17)
    x0 = K.rest_on_wall(x0, np.array([n]), mat.r)
    wall = K.wall_facet(mat, extent=200 * mat.r)

    def desc(total, precision):
        _, d = _desc(total, A.LG_BINARY_SINTER, A.LG_HAMAKER_LIMITED, A.LG_PAIRS_VERLET, A.LG_FORCE_KERNEL_COMPACT, precision,
                     max_neighbors=96, n_facets=1, facet_auto_move=1)
        return d

    sched = [(1, 20), (39, 20)]
    xs, vs, sizes = np.tile(x0, (count, 1)), np.tile(v0, (count, 1)), [n] * count
    a = _run(desc(n * count, A.LG_PRECISION_MIXED), xs, vs, sched, sizes=sizes, facets=[wall])
    b = _run(desc(n * count, A.LG_PRECISION_MIXED), xs, vs, sched, sizes=sizes, facets=[wall], graphs=False)
    _same(a, b)
    for f in a:
        for q in range(1, count):
            assert np.array_equal(f[q * n:(q + 1) * n], f[:n]), q
    ref = _run(desc(n, A.LG_PRECISION_FP64), x0, v0, [], facets=[wall])
    assert H.rel_err(a[0][:n], ref[0]) <= 1e-6


@pytest.mark.parametrize("precision", [A.LG_PRECISION_FP64, A.LG_PRECISION_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("m", [5, 7, 10])
def test_rows_that_outgrow_their_first_capacity(m, precision):
    """A cubic lattice at contact: 56 partners within 4.5 r, more than the 48 slots that rows start with. The handle
    moves to longer rows at its creation; it steps as one that was given them."""
    mat = K.Material()
    g = np.arange(m) * 2.0 * mat.r * 0.999
    x0 = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    v0 = generate_velocities(3, len(x0), 0.1)
    runs = []
    for cap in (0, 84):
        _, d = _desc(len(x0), A.LG_BINARY_CONTACT, A.LG_HAMAKER_LIMITED, A.LG_PAIRS_VERLET, A.LG_FORCE_KERNEL_AUTO, precision,
                     max_neighbors=cap)
        runs.append(_run(d, x0, v0, [(1, 0), (25, 10)]))
    _same(*runs)
