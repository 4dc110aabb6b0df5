"""pms without the column store (csrc/complex2.cu) against the oracle's twist,
at the sizes and forms where its kernels take another branch, and the inputs
it must leave to the general path."""
import numpy as np
import pytest

import oracle
from cases import lower_star_volume, random_complex, simplex_skeleton, triangle
from openph_gb300 import complexes as cx
from openph_gb300.complexes import BoundaryMatrix

pytestmark = pytest.mark.gpu


def check(ctx, bm, **kw):
    want, want_ess, _ = oracle.twist(bm)
    low, ess, arg, info = ctx.reduce(bm, "pms", with_arglow=True)
    np.testing.assert_array_equal(low, want)
    np.testing.assert_array_equal(ess, want_ess)
    want_arg = np.full(bm.m, -1, np.int32)
    want_arg[want[want >= 0]] = np.flatnonzero(want >= 0)
    np.testing.assert_array_equal(arg, want_arg)
    return info


def shuffled(bm, seed):
    """The same complex in another filtration order: a random value per
    simplex, at least its faces' (kinds of columns interleave freely)."""
    rng = np.random.default_rng(seed)
    val = rng.random(bm.m)
    for j in range(bm.m):
        col = bm.column(j)
        if len(col):
            val[j] = max(val[j], val[col].max() + 1e-9)
    order = np.argsort(val, kind="stable")
    pos = np.empty(bm.m, np.int64)
    pos[order] = np.arange(bm.m)
    return BoundaryMatrix.from_columns([sorted(pos[bm.column(j)].tolist()) for j in order])


def graph(n_vertices, edges):
    return BoundaryMatrix.from_columns([[] for _ in range(n_vertices)] + [sorted(e) for e in edges])


# one tile of columns is 2048; 24 x 14 is 1,909 columns, 21 x 17 is 2,029, 18 x 20 is 2,047, 19 x 19 2,053
@pytest.mark.parametrize("h,w,sigma", [(2, 2, 0.5), (2, 40, 1.0), (18, 20, 1.0), (19, 19, 0.5), (63, 65, 3.0),
                                       (97, 203, 4.0), (150, 160, 0.3)])
def test_images(ctx, h, w, sigma):
    assert check(ctx, cx.lower_star_image(h, w, seed=h + w, sigma=sigma))["sweeps"] >= 1


@pytest.mark.parametrize("kind", ["flat", "ties", "stairs", "bowl"])
def test_images_of_special_order(ctx, kind):
    y, x = np.mgrid[0:40, 0:37]
    img = {"flat": 0 * x, "ties": (7 * x * x + 5 * y) % 4, "stairs": (x % 2) * 100 - x,
           "bowl": (x - 15.2) ** 2 + 0.5 * (y - 20.1) ** 2}[kind]
    check(ctx, cx.lower_star(img.astype(np.float32)))


@pytest.mark.parametrize("seed", range(3))
def test_kinds_interleaved(ctx, seed):
    check(ctx, shuffled(cx.lower_star_image(20, 15, seed=seed, sigma=1.0), seed))


def test_graphs(ctx):
    rng = np.random.default_rng(5)
    path = [(i, i + 1) for i in range(299)]
    check(ctx, graph(300, path))
    check(ctx, graph(300, path[::-1]))  # every edge but the first joins a younger singleton
    check(ctx, graph(40, [(0, i) for i in range(1, 40)]))
    multi = [tuple(sorted(rng.choice(30, 2, replace=False).tolist())) for _ in range(200)]  # parallel edges
    check(ctx, graph(34, multi))
    check(ctx, graph(2, [(0, 1)]))


def test_batch_of_images_and_graphs(ctx):
    mats = [cx.lower_star_image(9, 12, seed=1, sigma=1.0), BoundaryMatrix.from_columns([]), graph(5, [(0, 4), (1, 2)]),
            BoundaryMatrix.from_columns([[]] * 3), cx.lower_star_image(31, 22, seed=2, sigma=1.0), triangle()]
    lows, esss, _ = ctx.reduce_batch(mats, "pms")
    for bm, low, ess in zip(mats, lows, esss):
        if bm.m:
            want, want_ess, _ = oracle.twist(bm)
            np.testing.assert_array_equal(low, want)
            np.testing.assert_array_equal(ess, want_ess)


def test_left_to_the_general_path(ctx):
    """Matrices that are no such complex give what 'never' (the sweeps on D)
    gives: a column of one row, of four rows, rows of the wrong kind, three
    edges that bound nothing, and larger complexes."""
    path3 = BoundaryMatrix.from_columns([[], [], [], [], [0, 1], [1, 2], [2, 3], [4, 5, 6]])
    one_row = BoundaryMatrix.from_columns([[], [], [0], [0, 1]])
    squares = BoundaryMatrix.from_columns([[], [], [], [], [0, 1], [1, 2], [2, 3], [0, 3], [4, 5, 6, 7]])
    mixed = BoundaryMatrix.from_columns([[], [], [], [0, 1], [0, 2], [1, 2], [3, 4, 5], [0, 1, 2]])
    edge_on_edge = BoundaryMatrix.from_columns([[], [], [0, 1], [0, 2]])
    for bm in (path3, one_row, squares, mixed, edge_on_edge, simplex_skeleton(7, seed=3), lower_star_volume(4, seed=1)):
        ctx.set_dual("never")
        low_n, ess_n, _ = ctx.reduce(bm, "pms")
        ctx.set_dual("auto")
        low, ess, _ = ctx.reduce(bm, "pms")
        np.testing.assert_array_equal(low, low_n)
        np.testing.assert_array_equal(ess, ess_n)


@pytest.mark.parametrize("p_tri", [0.1, 0.5])
def test_crowded_edges(ctx, p_tri):
    """Sparse 2-complexes, some of whose edges have more than two triangles."""
    for seed in range(4):
        check(ctx, random_complex(16, 0.4, p_tri, seed))


@pytest.mark.parametrize("n", [3, 4, 5, 31, 32, 33, 50, 65, 100])
def test_rips_full(ctx, n):
    check(ctx, cx.rips_cube(n, seed=n))
    check(ctx, cx.rips(cx.points_circle(n, seed=n)))


@pytest.mark.parametrize("target", [3_000, 40_000, 200_000, 700_000])
def test_rips_thresholds(ctx, target):
    """Torus complexes cut off early: essential classes, several components,
    windows of triangles left behind."""
    check(ctx, cx.rips_torus(300, target, seed=target))


def test_rips_ties(ctx):
    """Equal distances (a grid, repeated points): few apparent pairs."""
    g = np.stack(np.meshgrid(*[np.arange(3.0)] * 3), -1).reshape(-1, 3)
    check(ctx, cx.rips(g))
    check(ctx, cx.rips(g, threshold=1.5))
    check(ctx, cx.rips(np.repeat(g[:12], 3, axis=0)))


@pytest.mark.parametrize("n,seed", [(12, 0), (20, 1), (28, 2)])
def test_rips_in_any_order(ctx, n, seed):
    """Random filtration orders: most edges are residual, their columns sums
    of many, claimed and taken over by CTAs at the same time."""
    check(ctx, shuffled(cx.rips_cube(n, seed=seed), seed))


def test_doubled_simplices(ctx):
    """Two triangles on the same edges, two edges on the same vertices: no
    simplicial complex, and too many triangles for a graph."""
    tri = [[0, 1], [0, 2], [1, 2]]
    cols = [[], [], []] + tri + [[3, 4, 5]] * 4
    check(ctx, BoundaryMatrix.from_columns(cols))
    cols = [[], [], []] + tri + [[1, 2]] + [[3, 4, 5], [3, 4, 6], [3, 4, 5], [3, 4, 6], [3, 4, 6]]
    check(ctx, BoundaryMatrix.from_columns(cols))


def test_batch_of_rips(ctx):
    mats = [cx.rips_mixed(n, seed=70 + n) for n in (60, 3, 25, 2, 1, 40)]
    mats[2:2] = [BoundaryMatrix.from_columns([]), triangle(), cx.lower_star_image(9, 7, seed=5)]
    mats.append(shuffled(cx.rips_cube(18, seed=9), 4))
    lows, esss, _ = ctx.reduce_batch(mats, "pms")
    for bm, low, ess in zip(mats, lows, esss):
        if bm.m:
            want, want_ess, _ = oracle.twist(bm)
            np.testing.assert_array_equal(low, want)
            np.testing.assert_array_equal(ess, want_ess)


def test_runs_and_not(ctx):
    """Orders next to a Rips filtration's that the run form must refuse: a
    vertex between an edge and its triangle, the third vertices of an edge's
    triangles descending, an edge between an edge and its triangles."""
    tri = [[0, 1], [0, 2], [1, 2]]
    late = BoundaryMatrix.from_columns([[], [], []] + tri + [[], [3, 4, 5]])
    check(ctx, late)
    # edge (0, 1) last, with third vertices 2, 3 and 4
    cols = [[] for _ in range(5)] + [[0, v] for v in (2, 3, 4)] + [[1, v] for v in (2, 3, 4)] + [[0, 1]]
    runs = [[5, 8, 11], [6, 9, 11], [7, 10, 11]]
    for order in (runs, runs[::-1], [runs[1], runs[0], runs[2]]):
        check(ctx, BoundaryMatrix.from_columns(cols + order))
    check(ctx, BoundaryMatrix.from_columns(cols + [runs[0], [2, 3], runs[1], runs[2]]))


@pytest.mark.parametrize("n", [159, 160, 161, 164])
def test_rips_cta_sizes(ctx, n):
    """Either side of the residual columns' CTA and window sizes."""
    check(ctx, cx.rips(cx.points_circle(n, seed=n), threshold=1.2))


@pytest.mark.parametrize("points,threshold", [(cx.points_circle(165, 2), np.inf), (cx.points_cube(200, 3), np.inf),
                                              (cx.points_cube(1000, 4), 0.29), (cx.points_circle(190, 5), 1.7)])
def test_residual_windows(ctx, points, threshold):
    """Large complexes of several windows of 2^18 triangles: columns published
    with windows before, at and after those they are added in."""
    check(ctx, cx.rips(points, threshold))


@pytest.mark.parametrize("n_max", [100, 121, 125, 140])
def test_batch_of_whole_instances(ctx, n_max):
    """130 instances: a CTA each while every one fits its shared memory, the
    grid-wide kernels for the whole batch where one does not."""
    sizes = np.full(130, 6, np.int32)
    sizes[[3, 77]] = n_max, 65
    sizes[[8, 9]] = 1, 2
    seeds = np.arange(130, dtype=np.uint64) + np.uint64(5)
    col_off, colptr, rows = cx.rips_mixed_instances(sizes, seeds)
    low, ess, _ = ctx.reduce_batch_packed(col_off, colptr, rows)
    for b in range(130):
        bm = cx.batch_instance(col_off, colptr, rows, b)
        want, want_ess, _ = oracle.twist(bm)
        np.testing.assert_array_equal(low[col_off[b]:col_off[b + 1]], want, err_msg=str(b))
        np.testing.assert_array_equal(ess[col_off[b]:col_off[b + 1]], want_ess, err_msg=str(b))


@pytest.mark.parametrize("count,n,large,swap", [(1, 34, (34,), False), (1, 57, (57,), True), (9, 20, (48, 61), False),
                                                (150, 30, (90, 96, 97), False), (400, 34, (64, 65, 90), False),
                                                (400, 34, (64, 90), True)])
def test_batch_of_uneven_instances(ctx, count, n, large, swap):
    """Instances above and below their share of a CTA, fewer and more than
    CTAs: the larger ones in pieces, the largest first.  With two of the last
    one's triangles exchanged it is no complex in runs, and the batch goes to
    the general path."""
    sizes = np.full(count, n, np.int32)
    sizes[-len(large):] = large
    col_off, colptr, rows = cx.rips_mixed_instances(sizes, np.arange(count, dtype=np.uint64) + np.uint64(11))
    if swap:
        end = int(colptr[-1])
        rows = rows.copy()
        rows[end - 6:] = np.concatenate([rows[end - 3:], rows[end - 6:end - 3]])
    low, ess, _ = ctx.reduce_batch_packed(col_off, colptr, rows)
    mats = [cx.batch_instance(col_off, colptr, rows, b) for b in range(count)]
    for b in sorted({0, count // 3, *range(max(0, count - 5), count)}):
        want, want_ess, _ = oracle.twist(mats[b])
        np.testing.assert_array_equal(low[col_off[b]:col_off[b + 1]], want, err_msg=str(b))
        np.testing.assert_array_equal(ess[col_off[b]:col_off[b + 1]], want_ess, err_msg=str(b))


@pytest.mark.parametrize("cut", [1, 2, 3, 40, 300, 2000, 2300])
def test_first_simplices_of_a_rips_complex(ctx, cut):
    """A filtration cut off anywhere: inside the last edge's run, right after
    an edge, among the vertices."""
    bm = cx.rips_cube(24, seed=6)
    check(ctx, BoundaryMatrix(bm.colptr[:cut + 1], bm.rows[:bm.colptr[cut]]))
    big = cx.rips_cube(80, seed=6)
    cut = cut * 30
    check(ctx, BoundaryMatrix(big.colptr[:cut + 1], big.rows[:big.colptr[cut]]))


def test_missing_triangle(ctx):
    """Rips complexes less one triangle each: no flag complexes."""
    for n in (12, 70):
        bm = cx.rips_cube(n, seed=3)
        size = np.diff(bm.colptr)
        drop = np.flatnonzero(size == 3)[::max(1, bm.m // 7)]
        for t in drop:
            cols = np.delete(np.arange(bm.m), t)
            colptr = np.concatenate([[0], np.cumsum(size[cols])])
            rows = np.concatenate([bm.rows[:bm.colptr[t]], bm.rows[bm.colptr[t + 1]:]])
            check(ctx, BoundaryMatrix(colptr, rows - (rows > t)))
