"""Counts of the flat kernel far from the small launches of the other tests: closed
forms modulo 2^64, as the reference's unsigned 64-bit counters, and batches
whose results are copied back instead of written by the kernel."""
import random

import numpy as np
import pytest

from tests.golden.make_golden import random_pattern

pytestmark = pytest.mark.gpu

# two adjacent vertices and three common neighbours
BOOK = "".join(f"v {i} 1\n" for i in range(5)) + "e 0 1 1\n" + "".join(f"e {a} {b} 1\n" for b in (2, 3, 4) for a in (0, 1))


@pytest.mark.parametrize("pages", [3, 4, 5, 100, 3_000_001, 3_400_000, 3_400_001, 3_400_002])
def test_triples_of_a_large_set(T, pages):
    """Two adjacent hubs with `pages` common neighbours: 12 C(pages, 3) embeddings."""
    n = pages + 2
    rowptr = np.concatenate([[0, n - 1, 2 * (n - 1)], 2 * (n - 1) + 2 * np.arange(1, pages + 1)]).astype(np.int64)
    every = np.arange(n, dtype=np.int32)
    colidx = np.concatenate([every[1:], np.delete(every, 1), np.tile(np.array([0, 1], np.int32), pages)])
    G = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx)
    P = T.PatternPreprocessor(text=BOOK)
    assert P.dump()["flat"]["t"] == 3 and P.dump()["flat"]["form"] == 1
    assert T.count(G, P).count == 12 * (pages * (pages - 1) * (pages - 2) // 6) % 2 ** 64


@pytest.mark.parametrize("n", [511, 512, 513, 1500, 16384])
def test_results_of_large_batches(T, n):
    """Up to 512 slots the kernel writes the counts to the host, beyond they are copied."""
    G = T.GraphPreprocessor(csr=T.gen_er(1000, 10.0, 0).set_labels(5, 2), labeled=True)
    rng = random.Random(n)
    base = [T.PatternPreprocessor(text=random_pattern(3 + i % 3, 0.5, 5, rng), labeled=True) for i in range(101)]
    want = [T.count(G, p).count for p in base]
    plans = [base[i % 101] for i in range(n)]
    for opt in ({}, {"graph_capture": 1}, {"graph_capture": 1}):
        assert T.count_batch(G, plans, T.default_options(**opt))[0] == [want[i % 101] for i in range(n)]
        assert T.last_launch(G)["mean_warp_ms"] > 0


@pytest.mark.parametrize("warps", range(1, 9))
@pytest.mark.parametrize("cap", [64, 1024, 4096, 8192])
def test_the_deepest_buffers_that_are_accepted(T, warps, cap):
    """A depth that one kernel accepts the other accepts: buffers up to all of an SM's shared memory."""
    G = T.GraphPreprocessor(csr=T.gen_er(1000, 20.0, 0))
    for text in (BOOK, "".join(f"v {i} 1\n" for i in range(4)) + "e 0 1 1\ne 0 2 1\ne 1 2 1\ne 0 3 1\ne 1 3 1\ne 2 3 1\n"):
        P = T.PatternPreprocessor(text=text)
        want = T.count(G, P).count
        got = []
        for kernel in ({}, {"tail_count": 1}):
            try:
                got.append(T.count(G, P, T.default_options(warps_per_block=warps, chunk_cap=cap, **kernel)).count)
            except T.TdfsError as e:
                got.append(e.code)
        assert got in ([want, want], [5, 5]), (warps, cap)  # 5: TDFS_ERR_CAPACITY
