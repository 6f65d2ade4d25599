"""A graph's row membership tables are spare memory: where a launch workspace or
another graph's arrays find no room on the device, they are given up and the
counts go on with the DFS kernel."""
import ctypes as C
import gc

import numpy as np
import pytest

from tests.patterns import TRIANGLE, clique

pytestmark = pytest.mark.gpu

N, D = 100_000, 20  # every vertex is adjacent to the D before and the D after it, around a ring
MB = 1 << 20


def ring():
    steps = np.concatenate([np.arange(-D, 0), np.arange(1, D + 1)])
    rows = np.sort((np.arange(N)[:, None] + steps) % N, axis=1).astype(np.int32)
    triangles = N * sum(int(b - a in set(steps)) for a in steps for b in steps)
    return np.arange(N + 1, dtype=np.int64) * 2 * D, rows.ravel(), triangles


@pytest.fixture
def full(T):
    """Graphs that hold every pooled workspace, and a function that leaves so
    many bytes free on the device."""
    import torch
    held = []
    for _ in range(6):
        held.append(T.GraphPreprocessor(csr=T.gen_er(500, 8.0, 1)))
        for opt in ({}, {"tail_count": 1}):  # (either kernel is loaded)
            T.count(held[-1], T.PatternPreprocessor(text=TRIANGLE), T.default_options(**opt))
    ballast = []

    def leave(nbytes):
        gc.collect()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        ballast.append(torch.empty(free - nbytes, dtype=torch.uint8, device="cuda"))
        return torch.cuda.mem_get_info()[0]

    yield leave
    ballast.clear()
    torch.cuda.empty_cache()
    for g in held:
        g.close()


def sizes():
    tables = 32 * (N + N * 2 * D * 5 // 16 + 1)
    arrays = 2 * 4 * N * 2 * D + 12 * N
    return arrays, tables


def bytes_now(T, G):
    b = C.c_size_t()
    T.lib().tdfs_graph_info(G._h, None, None, None, None, C.byref(b))
    return b.value


def test_a_count_finds_room_for_its_workspace(T, full):
    rowptr, colidx, want = ring()
    arrays, tables = sizes()
    P = T.PatternPreprocessor(text=TRIANGLE)
    full(arrays + tables + 12 * MB)  # a workspace takes more than what the graph leaves of it
    G = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx)
    for _ in range(3):
        assert T.count(G, P).count == want
    assert bytes_now(T, G) == G.device_bytes - tables
    assert T.count_batch(G, [P, P])[0] == [want] * 2
    G.close()


def test_another_graph_finds_room_for_its_arrays(T, full):
    rowptr, colidx, want = ring()
    arrays, tables = sizes()
    P = T.PatternPreprocessor(text=TRIANGLE)
    full(arrays + tables + 64 * MB)
    G = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx)
    assert T.count(G, P).count == want and bytes_now(T, G) == G.device_bytes
    full(arrays - 10 * MB)  # not enough for the other graph
    H = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx)
    assert T.count(G, P).count == want and bytes_now(T, G) == G.device_bytes - tables
    G.close()
    assert T.count(H, P).count == want
    H.close()


def test_level_two_buffers_are_as_many_as_the_grid_has_warps(T, full):
    import torch
    csr = T.gen_chung_lu(30000, 90000, 2.1, 9000, 1)
    G = T.GraphPreprocessor(csr=csr)
    assert G.max_degree > 4096
    P = T.PatternPreprocessor(text=clique(5))
    part = dict(edge_end=400)

    def count(**kw):
        return T.count(G, P, T.default_options(**part, **kw)).count

    want = count(tail_count=1)  # the DFS kernel: the workspace is there, the buffers are not
    T.count(G, T.PatternPreprocessor(text=TRIANGLE))
    free = torch.cuda.mem_get_info()[0]
    assert want > 0 and count(blocks_per_sm=1) == want
    few = free - torch.cuda.mem_get_info()[0]
    assert count() == want
    assert 0 < few < free - torch.cuda.mem_get_info()[0] < 56 * MB
    # captured launches follow when the buffers grow and move
    for shape in ({}, {}, {"warps_per_block": 1}, {}, {"warps_per_block": 1}, {"blocks_per_sm": 1}, {}):
        for _ in range(3):
            assert count(graph_capture=1, **shape) == want
    G.close()
