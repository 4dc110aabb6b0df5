"""The server's lanes (2-complexes reduced beside the sweeps) and the sweeps at
work together: the limit on active requests, the switches that keep requests
on the sweeps, and budgets that some requests' lanes cannot hold."""
import threading

import numpy as np
import pytest

import oracle
from cases import lower_star_volume
from openph_gb300 import complexes as cx
from openph_gb300.api import Server

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mix():
    """Complexes that the lanes take and volumes that they pass on."""
    reqs = []
    for s in range(6):
        reqs += [lower_star_volume(5 + s % 3, seed=s), cx.rips_cube(20 + 8 * s, seed=s),
                 cx.lower_star_image(30 + 17 * s, 40, seed=s, sigma=2.0), cx.rips_torus(90, 20_000, seed=s)]
    return reqs, [oracle.twist(bm)[:2] for bm in reqs]


def check(srv, tickets, want):
    for t, (low, ess) in zip(tickets, want):
        got_low, got_ess, _ = srv.wait(t)
        np.testing.assert_array_equal(got_low, low)
        np.testing.assert_array_equal(got_ess, ess)


@pytest.mark.parametrize("max_active", [1, 2, 4, 64])
def test_max_active(cuda_lib, mix, max_active):
    """No more requests at work than the limit, lanes included, whatever comes
    first; and all of them done."""
    reqs, want = mix
    seen, stop = [], threading.Event()
    with Server(0, budget_bytes=2 << 30, max_active=max_active) as srv:
        def watch():
            while not stop.is_set():
                seen.append(srv.stats()["active"])
        th = threading.Thread(target=watch)
        th.start()
        try:
            for order in (range(len(reqs)), reversed(range(len(reqs)))):
                order = list(order)
                check(srv, [srv.submit(reqs[k]) for k in order], [want[k] for k in order])
        finally:
            stop.set()
            th.join()
        assert srv.stats()["completed"] == 2 * len(reqs)
    assert 1 <= max(seen) <= max_active


@pytest.mark.parametrize("switch", [None, "OPH_SERVE_CHAIN_CAP", "OPH_NO_CLUSTER", "OPH_NO_INST_TRANSPOSE",
                                    "OPH_HOST_LOOP", "OPH_TRACE"])
def test_switches_of_the_general_path(cuda_lib, monkeypatch, mix, switch):
    """Without one, 2-complexes take no sweep; with one set at creation, every
    request goes through the sweeps."""
    if switch:
        monkeypatch.setenv(switch, "0" if switch == "OPH_TRACE" else "1")
    reqs, want = mix
    lanes = [k for k in range(len(reqs)) if k % 4]
    with Server(0, budget_bytes=8 << 30, max_active=8) as srv:
        check(srv, [srv.submit(reqs[k]) for k in lanes], [want[k] for k in lanes])
        assert (srv.stats()["sweeps"] > 0) == bool(switch)


@pytest.mark.parametrize("budget", [64 << 20, 256 << 20, 2 << 30])
def test_requests_beyond_a_lane(cuda_lib, mix, budget):
    """Budgets whose lanes hold some of the requests, or next to none: those go
    to the sweeps, beside the lanes."""
    reqs, want = mix
    with Server(0, budget_bytes=budget, max_active=16) as srv:
        for _ in range(2):
            check(srv, [srv.submit(bm) for bm in reqs], want)
        assert srv.stats()["sweeps"] > 0 and srv.stats()["completed"] == 2 * len(reqs)


@pytest.mark.parametrize("max_active", [2, 3, 4])
def test_admissions_beside_a_last_sweep(cuda_lib, mix, max_active):
    """Few places: a sweep often finds every listed request reduced while others
    are being admitted, into columns that earlier ones have left."""
    reqs, want = mix
    order = [k for k in range(len(reqs)) if k % 4 == 0] * 3  # the volumes, which need sweeps
    for _ in range(25):
        with Server(0, budget_bytes=1 << 30, max_active=max_active) as srv:
            check(srv, [srv.submit(reqs[k]) for k in order], [want[k] for k in order])
