"""What pms without the column store (csrc/complex2.cu) may take, and what it
must leave to the general path: matrices on either side of each check, through
every entry point that tries it, against the oracle's twist."""
import numpy as np
import pytest

import oracle
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
