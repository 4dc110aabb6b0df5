"""What pms without the column store (csrc/complex2.cu) may take, and what it
must leave to the general path: matrices on either side of each check, through
every entry point that tries it, against the oracle's twist."""
import numpy as np
import pytest

import oracle
from openph_gb300 import api
from openph_gb300 import complexes as cx
from openph_gb300.complexes import BoundaryMatrix

pytestmark = pytest.mark.gpu


def swapped(bm, edge):
    """The first two triangles of a run exchanged, in the first run of at
    least two from the edge of that number on."""
    size = np.diff(bm.colptr)
    edges = np.flatnonzero(size == 2)
    j = next(int(e) for e in edges[edge:] if e + 2 < bm.m and size[e + 1] == size[e + 2] == 3)
    rows, at = bm.rows.copy(), int(bm.colptr[j + 1])
    rows[at:at + 6] = np.concatenate([rows[at + 3:at + 6], rows[at:at + 3]])
    return BoundaryMatrix(bm.colptr, rows)


@pytest.mark.parametrize("n", [60, 80])
def test_refused_by_one_block_while_others_start(ctx, n):
    """A run found wrong among the first ones checked, when blocks of the same
    launch are still to begin: grid-wide, and in pieces of a batch's larger
    instances."""
    bm = swapped(cx.rips_cube(n, seed=n), 20)
    want, want_ess, _ = oracle.twist(bm)
    small = cx.rips_cube(30, seed=1)
    small_want, small_ess, _ = oracle.twist(small)
    for _ in range(3):
        low, ess, _ = ctx.reduce(bm, "pms")
        np.testing.assert_array_equal(low, want)
        np.testing.assert_array_equal(ess, want_ess)
        lows, esss, _ = ctx.reduce_batch([small] * 100 + [bm] * 50, "pms")
        for b in (0, 99, 100, 149):
            np.testing.assert_array_equal(lows[b], want if b >= 100 else small_want)
            np.testing.assert_array_equal(esss[b], want_ess if b >= 100 else small_ess)


@pytest.fixture(scope="module")
def server(cuda_lib):
    with api.Server(0, budget_bytes=4 << 30, max_active=64) as srv:
        yield srv


def device(bm):
    import torch
    return (torch.from_numpy(bm.colptr).cuda(), torch.from_numpy(bm.rows if bm.nnz else np.zeros(1, np.int32)).cuda(),
            torch.empty(2 * bm.m, dtype=torch.int32, device="cuda"))


def general(ctx, bm):
    """What the sweeps on D give, for matrices that are no complexes (twist
    leaves columns of one row alone, and clears by dimension)."""
    ctx.set_dual("never")
    low, ess, _ = ctx.reduce(bm, "pms")
    ctx.set_dual("auto")
    return low, ess


def check_everywhere(ctx, server, bm, batches=(3, 130), want=None):
    """Every entry point that tries the forms gives the oracle's lows: single
    calls with host and device input, with and without ess, 1-based, batches
    that take whole instances and that do not, and the server."""
    import torch
    want, want_ess = want or oracle.twist(bm)[:2]

    def same(low, ess, where):
        np.testing.assert_array_equal(low, want, err_msg=where)
        if ess is not None:
            np.testing.assert_array_equal(ess, want_ess, err_msg=where)

    low, ess, arg, _ = ctx.reduce(bm, "pms", with_arglow=True)
    same(low, ess, "host")
    want_arg = np.full(bm.m, -1, np.int32)
    want_arg[want[want >= 0]] = np.flatnonzero(want >= 0)
    np.testing.assert_array_equal(arg, want_arg)
    colptr, rows, out = device(bm)
    for with_ess in (True, False):
        torch.cuda.synchronize()
        ctx.reduce_device(bm.m, colptr.data_ptr(), rows.data_ptr(), out.data_ptr(),
                          out.data_ptr() + 4 * bm.m if with_ess else None)
        res = out.cpu().numpy()
        same(res[:bm.m], res[bm.m:] if with_ess else None, f"device, ess {with_ess}")
    r, c = bm.to_coo1()
    low, ess, *_ = api.ph("pms", r, c, bm.m)
    same(low - 1, ess, "ph")
    rips = cx.rips_cube(7, seed=2)
    rips_want, rips_ess, _ = oracle.twist(rips)
    for count in batches:
        mats = [rips] * (count - 1)
        mats.insert(count // 2, bm)
        lows, esss, _ = ctx.reduce_batch(mats, "pms")
        same(lows[count // 2], esss[count // 2], f"batch of {count}")
        for b in {0, count - 1} - {count // 2}:
            np.testing.assert_array_equal(lows[b], rips_want)
            np.testing.assert_array_equal(esss[b], rips_ess)
    low, ess, _ = server.wait(server.submit(bm))
    same(low, ess, "server")


def faces_late(bm, order):
    """The columns of bm, its simplices listed as `order` says."""
    pos = np.empty(bm.m, np.int64)
    pos[order] = np.arange(bm.m)
    return BoundaryMatrix.from_columns([sorted(pos[bm.column(j)].tolist()) for j in order])


# columns of three rows before the first edge, or without any edge: no run holds them
NO_EDGE_BEFORE = {
    "no edges": [[], [], [], [], [0, 1, 2], [0, 1, 3], [1, 2, 3]],
    "no edges, one": [[], [], [], [0, 1, 2]],
    "rows to the right": [[], [], [], [4, 5, 6], [0, 1], [0, 2], [1, 2]],
    "rows of vertices": [[], [], [], [0, 1, 2], [0, 1], [0, 2], [1, 2]],
    "one edge after": [[], [], [], [0, 1, 2], [0, 1]],
}


@pytest.mark.parametrize("name", NO_EDGE_BEFORE)
def test_three_rows_before_the_first_edge(ctx, server, name):
    check_everywhere(ctx, server, BoundaryMatrix.from_columns(NO_EDGE_BEFORE[name]))


@pytest.mark.parametrize("kind", ["rows to the right", "rows of vertices"])
def test_three_rows_before_the_first_edge_grid_wide(ctx, server, kind):
    """The same past 2^15 columns, where the runs are checked grid-wide."""
    bm = cx.rips_cube(60, seed=3)
    cols = [bm.column(j).tolist() for j in range(bm.m)]
    tri = [x + 1 for x in cols[next(j for j in range(bm.m) if len(cols[j]) == 3)]]
    cols = [[x + (x >= 60) for x in c] for c in cols]
    cols.insert(60, tri if kind == "rows to the right" else [0, 1, 2])
    check_everywhere(ctx, server, BoundaryMatrix.from_columns(cols), batches=(3,))


@pytest.mark.parametrize("row", [5, 7, -1])
def test_malformed_rows_before_the_first_edge(ctx, row):
    """Rows out of range in such a column are refused as anywhere else."""
    bm = BoundaryMatrix(np.array([0, 0, 0, 0, 3, 5]), np.array([0, 1, row, 0, 1], np.int32))
    low = np.empty(5, np.int32)
    colptr, rows, out = device(bm)
    import torch
    torch.cuda.synchronize()
    L = api.lib()
    assert L.oph_reduce(ctx.handle, api.algo_id("pms"), 5, bm.colptr, api._ptr(bm.rows), low, None, None,
                        None) == api.OPH_ERR_BAD_INPUT
    with pytest.raises(api.OphError) as e:
        ctx.reduce_device(5, colptr.data_ptr(), rows.data_ptr(), out.data_ptr())
    assert e.value.status == api.OPH_ERR_BAD_INPUT


# simplices of a complete complex (runs refused, edges crowded: the table), of an image (a graph), of three points
@pytest.mark.parametrize("make", [lambda: cx.rips_cube(30, seed=4), lambda: cx.rips_cube(62, seed=4),
                                  lambda: cx.lower_star_image(12, 15, seed=4), lambda: cx.rips_cube(3, seed=4)],
                         ids=["crowded", "crowded, large", "image", "triangle"])
@pytest.mark.parametrize("kinds", [(3, 0, 2), (0, 3, 2), (2, 0, 3), (3, 2, 0)])
def test_faces_after_cofaces(ctx, server, make, kinds):
    """Columns by their number of rows, triangles before edges or edges before
    vertices: rows above the diagonal are accepted input."""
    bm = make()
    size = np.diff(bm.colptr)
    order = np.concatenate([np.flatnonzero(size == k) for k in kinds])
    check_everywhere(ctx, server, faces_late(bm, order), batches=(3,) if bm.m > 30_000 else (3, 130))


def test_one_triangle_before_an_edge(ctx, server):
    """A Rips complex with some triangles moved before their last edge."""
    bm = cx.rips_cube(20, seed=5)
    size = np.diff(bm.colptr)
    rng = np.random.default_rng(6)
    key = np.arange(bm.m, dtype=float)
    for t in rng.choice(np.flatnonzero(size == 3), 12, replace=False):
        key[t] = bm.column(t).max() - 0.5 - 20 * rng.random()
    check_everywhere(ctx, server, faces_late(bm, np.argsort(key, kind="stable")))


def sparse(nv, cluster):
    """A complete complex on a few of nv vertices, the others alone."""
    bm = cx.rips_cube(cluster, seed=9)
    colptr = np.concatenate([np.zeros(nv - cluster, np.int64), bm.colptr])
    return BoundaryMatrix(colptr, bm.rows + np.int32(nv - cluster))


@pytest.mark.parametrize("nv", [1024, 1025, 8189, 8190, 8192, 8193])
@pytest.mark.parametrize("cluster", [5, 20])
def test_many_vertices(ctx, server, nv, cluster):
    """Either side of the forms' limits on vertices."""
    check_everywhere(ctx, server, sparse(nv, cluster), batches=(3,))


def reordered(bm, seed, only=None):
    """The complex in a random filtration order, or one in which the simplices
    of `only` rows take random values and the others their faces'."""
    rng = np.random.default_rng(seed)
    size = np.diff(bm.colptr)
    val = rng.random(bm.m)
    if only is not None:
        val[size != only] = 0
    for j in range(bm.m):
        col = bm.column(j)
        if len(col):
            val[j] = max(val[j], val[col].max() + (1e-9 if only in (None, len(col)) else 0))
    return faces_late(bm, np.argsort(val, kind="stable"))


@pytest.mark.parametrize("n,only", [(20, None), (36, None), (40, 2), (50, None), (62, None), (62, 2), (90, None)])
def test_random_orders(ctx, server, n, only):
    """Columns that are sums of sums, many claimed and taken over at the same
    time (up to and past the sizes of whole instances)."""
    check_everywhere(ctx, server, reordered(cx.rips_cube(n, seed=n), n, only), batches=(3,) if n > 50 else (3, 130))


def test_batches_with_one_that_no_form_takes(ctx):
    """First, in the middle and last in a batch: the CTAs stop at it, and the
    general path reduces the whole batch."""
    from cases import lower_star_volume, simplex_skeleton
    rips = [cx.rips_cube(20 + 7 * s % 40, seed=s) for s in range(140)]
    for odd in (lower_star_volume(3, seed=1), simplex_skeleton(7, seed=2),
                BoundaryMatrix.from_columns([[], [0], [], [0, 2]])):
        for at in (0, 70, 140):
            mats = rips[:at] + [odd] + rips[at:]
            lows, esss, _ = ctx.reduce_batch(mats, "pms")
            for b in {0, 1, at, 139, 140}:
                want, want_ess = general(ctx, odd) if b == at else oracle.twist(mats[b])[:2]
                np.testing.assert_array_equal(lows[b], want)
                np.testing.assert_array_equal(esss[b], want_ess)


@pytest.mark.parametrize("last", [0, 1, 2, 3, 4])
def test_last_columns_of_any_width(ctx, server, last):
    """The look at a host matrix's last columns: widths of other complexes at
    the end, before the last 64 columns, and at their edge."""
    bm = cx.rips_cube(9, seed=last)
    cols = [bm.column(j).tolist() for j in range(bm.m)]
    if last == 4:  # the triangles of four points
        points = []
        for j, c in enumerate(cols):
            points.append({j} if not c else set().union(*(points[x] for x in c)))
        rows = [j for j in range(bm.m) if len(cols[j]) == 3 and points[j] <= {0, 2, 3, 7}]
    else:
        rows = list(range(last))
    for gap in (0, 62, 63, 64, 200):
        m = BoundaryMatrix.from_columns(cols + [rows] + [[]] * gap)
        check_everywhere(ctx, server, m, batches=(3,), want=general(ctx, m))


@pytest.mark.parametrize("m", [1, 2, 3000, 70_000])
def test_vertices_only(ctx, server, m):
    """Nothing to reduce, through every entry point and algorithm."""
    bm = BoundaryMatrix(np.zeros(m + 1, np.int64), np.zeros(0, np.int32))
    check_everywhere(ctx, server, bm, batches=(3,))
    for algo in api.ALGORITHMS:
        low, ess, _ = ctx.reduce(bm, algo)
        assert (low == -1).all() and (ess == 1).all()


@pytest.mark.parametrize("points,cut", [(125, 262_015), (125, 262_016), (125, 262_017), (125, 325_625),
                                        (201, 1_310_592), (201, 1_310_593)])
def test_window_of_a_whole_instance(ctx, points, cut):
    """A grid's complex (ties: the table) cut off at the sizes of the residual
    columns' windows, alone and behind another in a batch."""
    g = np.stack(np.meshgrid(*[np.arange(6.0 if points > 125 else 5.0)] * 3), -1).reshape(-1, 3)[:points]
    bm = cx.rips(g)
    bm = BoundaryMatrix(bm.colptr[:cut + 1], bm.rows[:bm.colptr[cut]])
    want, want_ess, _ = oracle.twist(bm)
    low, ess, _ = ctx.reduce(bm, "pms")
    np.testing.assert_array_equal(low, want)
    np.testing.assert_array_equal(ess, want_ess)
    lows, esss, _ = ctx.reduce_batch([cx.rips_cube(9, seed=1), bm, cx.rips_cube(11, seed=1)], "pms")
    np.testing.assert_array_equal(lows[1], want)
    np.testing.assert_array_equal(esss[1], want_ess)
    np.testing.assert_array_equal(lows[2], oracle.twist(cx.rips_cube(11, seed=1))[0])


@pytest.mark.parametrize("n,only,copies", [(25, None, 6), (40, 2, 3), (60, None, 2), (30, 2, 50)])
def test_batches_in_random_order(ctx, n, only, copies):
    mats = [reordered(cx.rips_cube(n - k % 3, seed=k), 50 + k, only) for k in range(min(copies, 5))]
    want = [oracle.twist(bm)[:2] for bm in mats]
    order = [k % len(mats) for k in range(copies)]
    lows, esss, _ = ctx.reduce_batch([mats[k] for k in order], "pms")
    for k, low, ess in zip(order, lows, esss):
        np.testing.assert_array_equal(low, want[k][0])
        np.testing.assert_array_equal(ess, want[k][1])
