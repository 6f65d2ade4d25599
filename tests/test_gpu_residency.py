"""A count does not need its whole grid on the GPU at once.

A server's idle kernel holds one CTA on every SM for a few seconds (it leaves
by itself after idle_exit_ms); the counts beside it find room for part of
their CTAs only.  Those finish the count: no count runs out of its own, much
shorter, wait limit, and none waits for the server's kernel to leave."""
import time

import numpy as np
import pytest

from tests.patterns import HOUSE, TRIANGLE, clique

pytestmark = pytest.mark.gpu

HOLD_MS = 2000


@pytest.fixture(scope="module")
def beside(T):
    """Graphs, plans and expected counts, made before a server's kernel moves in."""
    import torch
    er, cl = T.gen_er(4096, 16.0, 0).set_labels(4, 2), T.gen_chung_lu(30000, 90000, 2.1, 9000, 1).set_labels(4, 2)
    graphs = [T.GraphPreprocessor(csr=c, labeled=True) for c in (er, cl)]
    lab = "v 0 1\nv 1 0\nv 2 2\nv 3 1\ne 0 1 1\ne 0 2 1\ne 1 2 1\ne 1 3 1\n"
    plans = [T.PatternPreprocessor(text=t) for t in (TRIANGLE, clique(4), clique(5))]
    plans += [T.PatternPreprocessor(text=HOUSE), T.PatternPreprocessor(text=lab, labeled=True)]
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (er.rowptr, er.colidx)]
    torch.cuda.synchronize()
    opts = [dict(edge_end=2000) if i == 3 else {} for i in range(len(plans))]

    def run(g, i, **kw):
        return T.count(graphs[g], plans[i], T.default_options(**opts[i], **kw)).count

    def static(i, **kw):
        return T.count_static(0, er.n, er.nedges, dev[0].data_ptr(), dev[1].data_ptr(), None, plans[i],
                              T.default_options(**opts[i], **kw))

    want = {(g, i): run(g, i) for g in range(2) for i in range(len(plans))}  # (loads every kernel)
    assert static(1) == want[0, 1]
    for _ in range(2):
        assert run(0, 1, graph_capture=1) == want[0, 1]
    return T.GraphPreprocessor(csr=er), plans[0], run, static, want


@pytest.mark.parametrize("shape", [{}, {"chunk_cap": 512}, {"warps_per_block": 1, "chunk_cap": 64}])
def test_counts_beside_a_resident_kernel(T, beside, shape):
    graph, triangle, run, static, want = beside
    srv = T.Server(graph, max_inflight=4, idle_exit_ms=HOLD_MS, blocks_per_sm=1, **shape)
    assert srv.wait(srv.submit(triangle))[0] == want[0, 0]  # its kernel is on the GPU from here
    for (g, i), n in want.items():
        assert run(g, i, wait_limit_ms=500) == n, (g, i)
        if g == 0 and i < 3:
            assert static(i, wait_limit_ms=500) == n
    assert run(0, 1, graph_capture=1, wait_limit_ms=500) == want[0, 1]
    srv.close()


@pytest.mark.parametrize("shape", [{}, {"chunk_cap": 128}, {"warps_per_block": 1, "chunk_cap": 64}, {"blocks_per_sm": 2}])
def test_a_limited_server_leaves_room_on_the_sm(T, beside, shape):
    graph, triangle, run, static, want = beside
    shape = {"blocks_per_sm": 1, **shape}
    for i in range(4):
        srv = T.Server(graph, max_inflight=4, idle_exit_ms=HOLD_MS, **shape)
        assert srv.wait(srv.submit(triangle))[0] == want[0, 0]
        t0 = time.monotonic()
        assert run(0, i) == want[0, i] and static(1) == want[0, 1]
        assert time.monotonic() - t0 < HOLD_MS / 2000, (shape, i)
        srv.close()
