"""The flat kernel's bounded wait runs out on the GPU, and what follows works.

The self-test ends with a launch of the flat kernel that nothing can complete
(no tickets, and a mailbox counted as full that nobody opens): its warps wait
to their bound, the last CTA writes the error to the host, and the next
launches, plain and captured, count as before."""
import pytest

from tests.patterns import CYCLE4, TRIANGLE, clique

pytestmark = pytest.mark.gpu

TIMEOUT = 6  # TDFS_ERR_TIMEOUT


def test_flat_wait_runs_out_to_its_bound(T):
    G = T.GraphPreprocessor(csr=T.gen_chung_lu(50000, 150000, 2.1, 3000, 1))
    plans = [T.PatternPreprocessor(text=t) for t in (TRIANGLE, CYCLE4, clique(4))]
    part = dict(edge_end=20000)
    want = T.count_batch(G, plans, T.default_options(**part))[0]
    warps = T.last_launch(G)["warps"]
    for _ in range(2):
        rc, ms = T.selftest_wait_limit(G, 300)
        assert rc == TIMEOUT and 299 <= ms < 3000
        st = T.last_launch(G)  # the flat kernel's: its warps did nothing but wait, all of the time
        assert st["warps"] >= warps and st["idle_fraction"] > 0.95 and 295 < st["mean_warp_ms"] < 3000
        for cap in (0, 1, 1, 1):
            assert T.count_batch(G, plans, T.default_options(graph_capture=cap, **part))[0] == want
    assert min(want) > 0
