"""A context's budget: what a call needs is found on a fresh context, and that
budget still suffices when other calls of the same context, or an attempt that
was given up, have left buffers behind."""
import numpy as np
import pytest

import oracle
from cases import lower_star_volume
from openph_gb300 import complexes as cx
from openph_gb300.api import OPH_ERR_OOM, Context, OphError

pytestmark = pytest.mark.gpu

GRAIN = 1 << 16
SMALL = 1 << 20  # what calls on small matrices may leave in buffers of their own (offsets, buckets)


def least(bm, algo, dual):
    """The least budget that a fresh context reduces bm with, to 64 KB."""
    def fits(nbytes):
        with Context(0) as c:
            c.set_budget(nbytes)
            c.set_dual(dual)
            try:
                c.reduce(bm, algo)
            except OphError as e:
                assert e.status == OPH_ERR_OOM
                return False
        return True

    lo, hi = 0, (1 << 32) // GRAIN
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid * GRAIN) else (mid, hi)
    return hi * GRAIN


def check(c, bm, algo):
    low, ess, _ = c.reduce(bm, algo)
    want, want_ess, _ = oracle.twist(bm)
    np.testing.assert_array_equal(low, want)
    if algo == "pms":
        np.testing.assert_array_equal(ess, want_ess)


@pytest.fixture(scope="module")
def volume():
    """No 2-complex: every attempt ends with the general path."""
    bm = lower_star_volume(9, seed=2)
    return bm, least(bm, "pms", "never")


def test_attempt_given_up(cuda_lib, volume):
    bm, need = volume
    with Context(0) as c:
        c.set_budget(need)
        check(c, bm, "pms")


@pytest.mark.parametrize("before", ["rips", "image", "batch", "generators", "ph_row"])
def test_buffers_of_other_calls(cuda_lib, volume, before):
    bm, need = volume
    with Context(0) as c:
        c.set_budget(need + SMALL)
        if before == "rips":
            c.reduce(cx.rips_cube(40, seed=1), "pms")
        elif before == "image":
            c.reduce(cx.lower_star_image(40, 40, seed=1), "pms")
        elif before == "batch":
            c.reduce_batch([cx.rips_cube(12, seed=s) for s in range(40)], "pms")
        elif before == "generators":
            cx.rips_device(cx.points_cube(500, seed=1), 0.3, ctx=c)
            cx.lower_star_device(cx.image_smoothed(200, 200, seed=1), ctx=c)
        else:
            check(c, cx.lower_star_image(40, 40, seed=1), "ph_row")
        for _ in range(2):
            check(c, bm, "pms")


def test_attempt_on_a_batch(cuda_lib):
    """The same for a batch, one of whose instances is no 2-complex."""
    mats = [cx.rips_cube(20, seed=s) for s in range(30)] + [lower_star_volume(4, seed=1)]
    want = [oracle.twist(bm) for bm in mats]

    def reduce(nbytes, dual):
        with Context(0) as c:
            c.set_budget(nbytes)
            c.set_dual(dual)
            return c.reduce_batch(mats, "pms")

    lo, hi = 0, (1 << 32) // GRAIN
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            reduce(mid * GRAIN, "never")
            hi = mid
        except OphError:
            lo = mid
    lows, esss, _ = reduce(hi * GRAIN, "auto")
    for (low, ess, _), a, b in zip(want, lows, esss):
        np.testing.assert_array_equal(a, low)
        np.testing.assert_array_equal(b, ess)


@pytest.mark.parametrize("algo", ["standard", "ph_row"])
def test_sequential_after_pms(cuda_lib, algo):
    bm = cx.lower_star_image(60, 60, seed=3)
    need = least(bm, algo, "auto")
    with Context(0) as c:
        c.set_budget(need + SMALL)
        check(c, cx.rips_cube(40, seed=1), "pms")
        for _ in range(2):
            check(c, bm, algo)


def test_large_generator_gives_its_scratch_back(cuda_lib):
    """The distances of 12,000 points (1.2 GB) are not kept by the context."""
    import torch
    with Context(0) as c:
        cx.rips_device(cx.points_cube(100, seed=1), 0.2, ctx=c)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        dm = cx.rips_device(cx.points_cube(12_000, seed=1), 0.01, ctx=c)
        del dm
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] > free - (1 << 28)
