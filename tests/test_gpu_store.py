"""The column store's own paths under the automatic choice.  Simplicial
2-complexes are reduced without the store now, so tests written for its
choices run here once more with a switch set that keeps calls on it (OPH_TRACE=0
traces nothing), and which way a matrix went is told by its kernel launches."""
import numpy as np
import pytest

import oracle
import test_gpu_dual
import test_gpu_inputs
import test_gpu_parity
import test_gpu_server
from cases import lower_star_volume
from openph_gb300 import complexes as cx
from openph_gb300.api import Context, Server
from openph_gb300.complexes import BoundaryMatrix
from test_gpu_acceptance import check_everywhere, reordered, server, sparse  # noqa: F401

pytestmark = pytest.mark.gpu
dctx, torus_1m, dual_mix = test_gpu_dual.dctx, test_gpu_parity.torus_1m, test_gpu_server.dual_mix


@pytest.fixture
def on_the_store(monkeypatch):
    monkeypatch.setenv("OPH_TRACE", "0")


@pytest.mark.parametrize("name", ["test_auto_choice", "test_dual_does_few_additions_on_rips",
                                  "test_rips_torus_1m_device_input"])
def test_automatic_choice(on_the_store, dctx, name):
    getattr(test_gpu_dual, name)(dctx)


def test_batch_auto(on_the_store, dctx):
    test_gpu_dual.test_batch(dctx, "auto")


def test_batch_transpose_both_ways(on_the_store, dctx, monkeypatch):
    test_gpu_dual.test_batch_transpose_both_ways(dctx, monkeypatch)


def test_calls_under_auto(on_the_store, cuda_lib, ctx, torus_1m):
    test_gpu_dual.test_drop_in_call_without_trackers(cuda_lib)
    test_gpu_parity.test_rips_torus_1m(cuda_lib, torus_1m, "auto")
    test_gpu_parity.test_batch_mixed(ctx)
    test_gpu_parity.test_batch_equals_alone(ctx)
    test_gpu_parity.test_batch_ragged_with_empty_instances(ctx)
    test_gpu_parity.test_context_reduce_arglow(ctx)
    test_gpu_parity.test_lower_star_512_full_size(ctx, "pms")
    test_gpu_inputs.test_batch_of_256_config_shaped_against_oracle(cuda_lib)


class Swept(Server):
    """A server all of whose requests must have gone through sweeps."""
    def submit(self, bm):
        t = super().submit(bm)
        self.requests = getattr(self, "requests", 0) + 1
        return t

    def wait(self, ticket, timeout_ms=-1):
        low, ess, info = super().wait(ticket, timeout_ms)
        assert info["sweeps"] > 0
        return low, ess, info

    def __exit__(self, *exc):
        if not exc[0]:
            st = self.stats()
            assert st["sweeps"] > 0 and st["completed"] >= getattr(self, "requests", 0) - 1
        super().__exit__(*exc)


@pytest.mark.parametrize("name", ["test_results_same_alone_and_in_the_mix", "test_arrivals_while_running",
                                  "test_request_larger_than_arena_is_rejected", "test_tight_arena_regrows",
                                  "test_device_submissions_mixed_with_host"])
def test_sweeps_of_the_server(on_the_store, cuda_lib, monkeypatch, name):
    monkeypatch.setattr(test_gpu_server, "Server", Swept)
    getattr(test_gpu_server, name)(cuda_lib)


@pytest.mark.parametrize("name", ["test_anti_transpose_requests_in_the_mix",
                                  "test_anti_transpose_requests_arriving_while_running",
                                  "test_anti_transpose_device_submission"])
def test_split_requests_of_the_server(on_the_store, cuda_lib, monkeypatch, dual_mix, name):
    monkeypatch.setattr(test_gpu_server, "Server", Swept)
    getattr(test_gpu_server, name)(cuda_lib, dual_mix)


def bipartite(n):
    """Every edge between two sets of n vertices: no triangles, more edges than the
    whole instances' first tables hold."""
    return BoundaryMatrix.from_columns([[]] * (2 * n) + [[u, n + v] for u in range(n) for v in range(n)])


# kernels launched: 2 for one instance of less than 6,144 columns (each time its tables were too small again), 4
# for a larger one, 6 for a graph, 7 for runs, 13 for the table after them, 9 where an instance was refused
FORMS = {
    "one instance": (lambda: cx.rips_cube(20, seed=1), 2),
    "one in pieces": (lambda: cx.rips_cube(40, seed=2), 4),
    "tables twice": (lambda: bipartite(60), 4),
    "graph": (lambda: cx.lower_star_image(90, 100, seed=3, sigma=2.0), 6),
    "graph after an instance": (lambda: cx.lower_star_image(20, 21, seed=4, sigma=1.0), 8),
    "runs, small CTAs": (lambda: cx.rips_cube(62, seed=5), 7),
    "runs, large CTAs": (lambda: cx.rips(cx.points_circle(170, 6), 1.0), 7),
    "table after an instance": (lambda: reordered(cx.rips_cube(20, seed=7), 7), 11),
    "table after the runs": (lambda: cx.rips(np.stack(np.meshgrid(*[np.arange(4.0)] * 3), -1).reshape(-1, 3)), 13),
    "table, many vertices": (lambda: sparse(5000, 20), None),
    "general": (lambda: lower_star_volume(5, seed=9), None),
}


@pytest.mark.parametrize("name", FORMS)
def test_which_form(cuda_lib, server, name):
    make, launches = FORMS[name]
    bm = make()
    want, want_ess, _ = oracle.twist(bm)
    with Context(0) as c:
        low, ess, _ = c.reduce(bm, "pms")
        got = c.last_profile()["kernel_launches"]
        np.testing.assert_array_equal(low, want)
        np.testing.assert_array_equal(ess, want_ess)
        if launches:
            assert got == launches
        elif name == "general":
            assert got > 20
        else:
            assert got < 20
        check_everywhere(c, server, bm, batches=(3,))


def test_whole_instances_twice(cuda_lib):
    """A batch whose edges exceed the first tables: once larger, and at once
    with the context's next call."""
    cycle = BoundaryMatrix.from_columns([[]] * 60 + [[v, v + 1] for v in range(59)] + [[0, 59]])
    mats = [cycle] * 200 + [cx.rips_cube(8, seed=1)]
    want = [oracle.twist(cycle)[:2], oracle.twist(mats[-1])[:2]]
    with Context(0) as c:
        for launches in (6, 3):
            lows, esss, _ = c.reduce_batch(mats, "pms")
            assert c.last_profile()["kernel_launches"] == launches
            for b in (0, 77, 199, 200):
                np.testing.assert_array_equal(lows[b], want[b == 200][0])
                np.testing.assert_array_equal(esss[b], want[b == 200][1])
