"""A graph's row membership tables are spare memory: where a launch workspace or
another graph's arrays find no room on the device, they are given up and the
counts go on with the DFS kernel."""
import ctypes as C
import gc

import numpy as np
import pytest

from tests.patterns import TRIANGLE

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
