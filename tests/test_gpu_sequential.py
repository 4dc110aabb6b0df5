"""The standard, twist and row algorithms with their columns side by side
(csrc/variants.cu, k_claim) against the oracle, where that takes another
branch: fewer columns than warps and more, more rows than a warp's bitmap
holds (73,728) and columns wider than its lists (768), a store that runs out,
and matrices whose order twist has to walk."""
import numpy as np
import pytest

import oracle
from cases import random_complex, simplex_skeleton, triangle
from openph_gb300.api import Context
from openph_gb300 import complexes as cx
from openph_gb300.complexes import BoundaryMatrix

pytestmark = pytest.mark.gpu

SHAPES = {
    "triangle": triangle,
    "cube": lambda: cx.rips_cube(17, seed=3),
    "skeleton": lambda: simplex_skeleton(8, seed=2),
    "random": lambda: random_complex(30, 0.5, 0.5, seed=5),
    "image": lambda: cx.lower_star_image(60, 71, seed=4, sigma=0.5),
    "smooth": lambda: cx.lower_star_image(45, 90, seed=6, sigma=6.0),
    "large": lambda: cx.lower_star_image(110, 113, seed=4, sigma=2.0),
    "circle": lambda: cx.rips(cx.points_circle(25, 2), np.inf),
}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("algo", ["standard", "twist", "ph_row_parallel"])
@pytest.mark.parametrize("pool", [0, 1])
def test_side_by_side(cuda_lib, shape, algo, pool):
    bm = SHAPES[shape]()
    with Context(0) as c:
        if pool:
            c.set_limits(initial_pool_bytes=pool)
        low, ess, info = c.reduce(bm, algo)
    want, want_ess, _ = oracle.twist(bm)
    np.testing.assert_array_equal(low, want)
    if algo != "ph_row_parallel":
        np.testing.assert_array_equal(ess, want_ess)


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("algo", ["standard", "twist"])
def test_any_matrix(ctx, seed, algo):
    """Columns that are no complex's boundaries: rows of several dimensions,
    above the diagonal too, so that what twist clears depends on its order."""
    rng = np.random.default_rng(seed)
    m = 150
    cols = [sorted(rng.choice(m, size=rng.integers(0, 6), replace=False).tolist()) for _ in range(m)]
    bm = BoundaryMatrix.from_columns(cols)
    low, *_ = ctx.reduce(bm, algo)
    np.testing.assert_array_equal(low, plain(cols, algo))


def plain(cols, algo):
    """The algorithm by its definition, on sets."""
    m = len(cols)
    work = [set(c) for c in cols]
    low = [max(c, default=-1) for c in work]
    holder = {}
    dims = [len(c) - 1 for c in cols]
    order = range(m)
    if algo == "twist":
        order = [j for d in range(max(dims), 0, -1) for j in range(m) if dims[j] == d]
    for j in order:
        while low[j] >= 0 and low[j] in holder:
            work[j] ^= work[holder[low[j]]]
            low[j] = max(work[j], default=-1)
        if low[j] >= 0:
            holder[low[j]] = j
            if algo == "twist":
                low[low[j]] = -1
    return np.array(low, np.int32)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("pool", [0, 1])
def test_row_estimate(cuda_lib, shape, pool):
    """The CPU row form's running essential estimate, replayed side by side."""
    bm = SHAPES[shape]()
    want, want_ess, st = oracle.ph_row(bm)
    with Context(0) as c:
        if pool:
            c.set_limits(initial_pool_bytes=pool)
        low, ess, info = c.reduce(bm, "ph_row")
    np.testing.assert_array_equal(low, want)
    np.testing.assert_array_equal(ess, want_ess)
    assert info["additions"] == st["additions"]


@pytest.mark.parametrize("seed", range(6))
def test_row_estimate_of_any_matrix(ctx, seed):
    """The same on columns that are no complex's boundaries, among them many
    with equal lows (the oracle's row form adds within one dimension only, so
    the walk over all columns is restated here)."""
    rng = np.random.default_rng(seed)
    m, rows = 150, (150, 20)[seed % 2]
    cols = [sorted(rng.choice(min(rows, max(j, 1)), size=min(int(rng.integers(0, 6)), j), replace=False).tolist())
            for j in range(m)]
    bm = BoundaryMatrix.from_columns(cols)
    want, want_ess = plain_row(cols)
    low, ess, _ = ctx.reduce(bm, "ph_row")
    np.testing.assert_array_equal(low, want)
    np.testing.assert_array_equal(ess, want_ess)


def plain_row(cols):
    """Rows from the bottom: the first column with the row as its low into the
    others; the estimate cleared at the row and the first column, and at a
    column that is then the first ever to hold its new low, and at that low; at the
    end at every pair (ph_row.cu:2-121)."""
    m = len(cols)
    work = [set(c) for c in cols]
    low = [max(c, default=-1) for c in work]
    first = [min((j for j in range(m) if low[j] == r), default=m) for r in range(m)]
    ess = [1] * m
    for i in range(m - 1, -1, -1):
        here = [j for j in range(m) if low[j] == i]
        if len(here) < 2:
            continue
        ess[i] = ess[here[0]] = 0
        for j in here[1:]:
            work[j] ^= work[here[0]]
            low[j] = max(work[j], default=-1)
            if low[j] >= 0:
                first[low[j]] = min(first[low[j]], j)
        for j in here[1:]:
            if low[j] >= 0 and first[low[j]] == j:
                ess[j] = ess[low[j]] = 0
    for j in range(m):
        if low[j] >= 0:
            ess[j] = ess[low[j]] = 0
    return np.array(low, np.int32), np.array(ess, np.int32)
