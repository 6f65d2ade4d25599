"""The flat kernel at the sizes where it can go wrong: buffers that refill after
every step, single-warp CTAs, one ticket per edge, work given away at once,
hub rows whose membership tables overflow buckets, rows of 0, 1, 7, 8 and 9
entries (the bucket size), self-loops, one-directional rows, label segments
and whole rows with labels, more labels than segments.  Counts are exact and
equal the oracle's."""
import random

import numpy as np
import pytest

from tests.golden.make_golden import random_pattern
from tests.patterns import CYCLE4, HOUSE, TRIANGLE, clique

pytestmark = pytest.mark.gpu

DIAMOND = "v 0 1\nv 1 1\nv 2 1\nv 3 1\ne 0 1 1\ne 0 2 1\ne 0 3 1\ne 1 2 1\ne 1 3 1\n"


def csr(edges, n):
    rows = [[] for _ in range(n)]
    for a, b in sorted(edges):
        rows[a].append(b)
    return (np.array([0] + list(np.cumsum([len(r) for r in rows])), np.int64),
            np.array([x for r in rows for x in r], np.int32))


def edge_graph():
    """Rows of 0..9 entries, two hubs adjacent to most vertices, self-loops and
    some one-directional edges."""
    n, rng, e = 900, random.Random(5), set()
    for v in range(2, n):
        for w in rng.sample(range(2, n), v % 10):
            e.add((v, w))
            if v % 3:
                e.add((w, v))
    for v in range(2, n - 20):
        e |= {(0, v), (v, 0)}
        if v % 2:
            e |= {(1, v), (v, 1)}
    e |= {(0, 1), (1, 0)} | {(v, v) for v in range(0, n, 7)}
    e = {(a, b) for a, b in e if a < n - 3}  # three empty rows
    return csr(e, n)


OPTIONS = [{}, {"chunk_cap": 64, "split_after_us": -1}, {"warps_per_block": 1, "blocks_per_sm": 1},
           {"edge_chunk": 1, "split_after_us": 1}, {"edge_chunk": 32, "warps_per_block": 3}, {"label_rows": -1},
           {"label_index": -1, "chunk_cap": 96}, {"graph_capture": 1}]


@pytest.fixture(scope="module")
def cases(T, po):
    rowptr, colidx = edge_graph()
    rng = random.Random(8)
    out = []
    for nlabels in (3, 20):  # label segments; more labels than segments
        labels = np.array([rng.randrange(nlabels) % 5 if nlabels > 16 else rng.randrange(nlabels)
                           for _ in range(len(rowptr) - 1)], np.int32)
        labels[0] = nlabels - 1
        out.append((T.GraphPreprocessor(rowptr=rowptr, colidx=colidx, labels=labels, labeled=True),
                    po.Graph(rowptr.copy(), colidx.copy(), labels.copy()), nlabels))
    return out


@pytest.mark.parametrize("opt", OPTIONS)
def test_edges_of_the_flat_kernel(T, po, cases, opt):
    rng = random.Random(4)
    texts = [(t, False) for t in (TRIANGLE, CYCLE4, DIAMOND, clique(4), clique(5))]
    texts += [(random_pattern(3 + i % 4, 0.3 + 0.1 * (i % 3), 3, rng), True) for i in range(12)]
    for dev, ora, nlabels in cases:
        for text, labeled in texts:
            if nlabels > 16 and not labeled:
                continue
            P = T.PatternPreprocessor(text=text, labeled=labeled)
            got = T.count(dev, P, T.default_options(**opt)).count
            assert got == po.count(ora, po.Plan(text, labeled)), (nlabels, text, labeled, opt)


@pytest.mark.parametrize("n", [1, 33, 200])
def test_many_plans_in_one_launch(T, cases, n):
    """Tickets run over all slots of a launch (a warp finds a ticket's slot 32 at
    a time); slots without tickets lie between the others."""
    dev, _, _ = cases[0]
    rng = random.Random(n)
    plans = [T.PatternPreprocessor(text=random_pattern(3 + i % 3, 0.5, 4, rng), labeled=True) for i in range(n)]
    assert T.count_batch(dev, plans)[0] == [T.count(dev, p).count for p in plans]


def test_flat_and_dfs_kernels_agree_on_a_power_law_graph(T):
    g = T.gen_chung_lu(30000, 90000, 2.1, 2500, 3).set_labels(3, 1)
    dev = T.GraphPreprocessor(csr=g, labeled=True)
    rng = random.Random(2)
    texts = [(t, False) for t in (TRIANGLE, CYCLE4, DIAMOND, clique(4), clique(5))]
    texts += [(random_pattern(4 + i % 2, 0.6, 3, rng), True) for i in range(4)]
    for text, labeled in texts:
        P = T.PatternPreprocessor(text=text, labeled=labeled)
        want = T.count(dev, P, T.default_options(tail_count=1)).count  # a DFS kernel knob: that kernel
        assert T.count(dev, P).count == want
        shards = [T.count(dev, P, T.shard_options(r, 3)).count for r in range(3)]
        assert sum(shards) == want


def test_level_two_in_global_memory(T):
    """On graphs with hubs of more than 4096 neighbours, plans that extend a
    vertex from its siblings keep level 2 in global memory, refilled when a
    candidate set outgrows it, and give children away as ranges."""
    n, hubs = 7000, 24
    rng = np.random.default_rng(6)
    e = set()
    for h in range(hubs):  # hubs adjacent to each other and to most vertices: sets beyond 2048 entries
        e |= {(h, int(v)) for v in rng.choice(n, 5200, replace=False) if v > h}
    e |= {(int(a), int(b)) for a, b in rng.integers(hubs, n, (9000, 2)) if a < b}
    e |= {(b, a) for a, b in e}
    rowptr, colidx = csr(e, n)
    labels = (np.arange(n) % 2).astype(np.int32)
    dev = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx, labels=labels, labeled=True)
    assert dev.max_degree > 4096
    # labeled: the same set reused by two later vertices
    fan = "".join(f"v {i} {int(i > 1)}\n" for i in range(5)) + "".join(
        f"e {a} {b} 1\n" for a, b in ((0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (2, 3), (3, 4)))
    for text, labeled in ((clique(4), False), (clique(5), False), (DIAMOND, False), (fan, True)):
        P = T.PatternPreprocessor(text=text, labeled=labeled)
        want = T.count(dev, P, T.default_options(tail_count=1)).count  # the DFS kernel
        assert want > 0
        for opt in ({}, {"split_after_us": -1, "edge_chunk": 1}, {"warps_per_block": 2, "chunk_cap": 64}):
            assert T.count(dev, P, T.default_options(**opt)).count == want, (text, opt)


def test_rows_that_break_the_rules_are_refused(T):
    """The CSR's rules, checked on the device: the error and what it says are
    those of the host's check, at the edges of rows, blocks and the arrays."""
    rowptr, colidx = edge_graph()
    n, E = len(rowptr) - 1, len(colidx)
    good = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx)
    assert good.max_degree == int(np.diff(rowptr).max())
    rows = [v for v in range(n) if rowptr[v + 1] - rowptr[v] >= 2]
    for v in (rows[0], rows[len(rows) // 2], rows[-1]):
        b, e = int(rowptr[v]), int(rowptr[v + 1])
        for at, val, what in ((b, -1, "out of range"), (e - 1, n, "out of range"), (b + 1, colidx[b], "strictly increasing")):
            c = colidx.copy()
            c[at] = val
            with pytest.raises(T.TdfsError) as ei:
                T.GraphPreprocessor(rowptr=rowptr, colidx=c)
            assert ei.value.code == 2 and what in str(ei.value) and f"row {v}" in str(ei.value)
        r = rowptr.copy()
        r[v + 1] = r[v] - 1 if r[v] else E + 5
        with pytest.raises(T.TdfsError) as ei:
            T.GraphPreprocessor(rowptr=r, colidx=colidx)
        assert ei.value.code == 2 and "rowptr decreases" in str(ei.value)
    for bad in (rowptr[:-1], rowptr + 1):  # the ends do not span the edges
        with pytest.raises(T.TdfsError) as ei:
            T.GraphPreprocessor(rowptr=bad, colidx=colidx)
        assert ei.value.code == 2


@pytest.mark.parametrize("nlabels", [1, 4, 16])
def test_long_rows_are_split_over_a_block(T, po, nlabels):
    """Rows around the length from which a whole CTA takes them (512) and far
    beyond: sources, neighbour degrees, tables and label segments, through
    the counts that use them."""
    n, rng, e = 3000, np.random.default_rng(nlabels), set()
    for h, d in enumerate((511, 512, 513, 1024, 2600)):
        for v in rng.choice(np.arange(10, n), d, replace=False):
            e |= {(h, int(v)), (int(v), h)}
    for a, b in rng.integers(5, n, (4000, 2)):
        if a != b:
            e |= {(int(a), int(b)), (int(b), int(a))}
    rowptr, colidx = csr(e, n)
    labels = rng.integers(0, nlabels, n).astype(np.int32)
    labels[0] = nlabels - 1
    dev = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx, labels=labels, labeled=True)
    ora = po.Graph(rowptr.copy(), colidx.copy(), labels.copy())
    r = random.Random(nlabels)
    for text, labeled in [(TRIANGLE, False), (CYCLE4, False)] + [(random_pattern(3 + i % 3, 0.5, nlabels, r), True)
                                                                for i in range(5)]:
        P = T.PatternPreprocessor(text=text, labeled=labeled)
        assert T.count(dev, P).count == po.count(ora, po.Plan(text, labeled)), (text, labeled)


@pytest.mark.parametrize("d", [127, 128, 129, 4095, 4097])
def test_tail_blocks_end_at_a_span_of_lists(T, d):
    """A block of a tail ends before its lists pass 4096 positions: 32 lists of
    128 fill it, the 32nd of 129 starts the next, one of 4097 is a block."""
    b = 8  # a clique of b vertices, each adjacent to all others: rows of d entries
    n = d + 1
    e = {(i, j) for i in range(b) for j in range(n) if i != j}
    rowptr, colidx = csr(e | {(j, i) for i, j in e}, n)
    labels = (np.arange(n) % 2).astype(np.int32)
    dev = T.GraphPreprocessor(rowptr=rowptr, colidx=colidx, labels=labels, labeled=True)
    edges = ("01 02 12 13 23 14 24", "01 02 03 04 12 13 14 23")
    for es in edges:
        for lab in ("11111", "01010", "11001"):
            text = "".join(f"v {i} {l}\n" for i, l in enumerate(lab)) + "".join(
                f"e {x[0]} {x[1]} 1\n" for x in es.split())
            P = T.PatternPreprocessor(text=text, labeled=lab != "11111")
            want = T.count(dev, P, T.default_options(tail_count=1)).count  # a DFS kernel knob: that kernel
            assert T.count(dev, P).count == want
            assert T.count(dev, P, T.default_options(split_after_us=-1)).count == want
