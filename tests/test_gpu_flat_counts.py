"""Counts of the flat kernel's closed forms far from the small graphs of the other
tests: modulo 2^64, as the reference's unsigned 64-bit counters."""
import numpy as np
import pytest

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
