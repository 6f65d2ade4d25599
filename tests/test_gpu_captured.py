"""Captured launches are made at a shape's first launch and kept with the launch
workspace, which passes from one data graph to the next: every replay counts
on the graph it was asked for, and no later call pays for the capture."""
import random
import statistics
import time

import pytest

from tests.golden.make_golden import random_pattern
from tests.patterns import CYCLE4, TRIANGLE, clique

pytestmark = pytest.mark.gpu


def plans(T, n, labels, seed):
    rng = random.Random(seed)
    named = [T.PatternPreprocessor(text=t) for t in (TRIANGLE, CYCLE4, clique(4))]
    return named + [T.PatternPreprocessor(text=random_pattern(3 + i % 4, 0.4, labels, rng), labeled=True)
                    for i in range(n)]


@pytest.mark.parametrize("kernel", [{}, {"tail_count": 1}, {"work_budget": 10 ** 12}])
def test_replays_follow_the_data_graph(T, kernel):
    csrs = [T.gen_er(1500 + 700 * i, 12.0, i).set_labels(3 + i % 2, i) for i in range(3)]
    csrs.append(T.gen_chung_lu(20000, 60000, 2.1, 5000, 4).set_labels(20, 1))
    plain, captured = T.default_options(**kernel), T.default_options(graph_capture=1, **kernel)
    P = plans(T, 3, 3, 1)
    graphs = [T.GraphPreprocessor(csr=c, labeled=True) for c in csrs]
    want = [T.count_batch(g, P, plain)[0] for g in graphs]
    for g in graphs:
        g.close()
    assert len({tuple(w) for w in want}) == len(want)
    for order in ([0, 1, 2, 3], [3, 0, 0, 2], [1, 3, 1, 2]):
        for i in order:  # one at a time: the workspace passes on
            g = T.GraphPreprocessor(csr=csrs[i], labeled=True)
            for _ in range(2):
                assert T.count_batch(g, P, captured)[0] == want[i]
            assert [T.count(g, p, captured).count for p in P] == want[i]
            g.close()
        graphs = [T.GraphPreprocessor(csr=csrs[i], labeled=True) for i in order]  # all at once
        for _ in range(2):
            for i, g in zip(order, graphs):
                assert T.count_batch(g, P, captured)[0] == want[i]
        for g in graphs:
            g.close()


def test_more_shapes_than_are_kept(T):
    g = T.GraphPreprocessor(csr=T.gen_er(1500, 12.0, 3).set_labels(4, 1), labeled=True)
    P = plans(T, 90, 4, 2)[3:]
    want = T.count_batch(g, P)[0]
    for _ in range(2):
        for n in range(1, len(P) + 1):  # a shape each
            assert T.count_batch(g, P[:n], T.default_options(graph_capture=1))[0] == want[:n]


def test_the_first_launch_of_a_shape_captures_it(T):
    g = T.GraphPreprocessor(csr=T.gen_er(2000, 12.0, 3))
    p = T.PatternPreprocessor(text=TRIANGLE)
    T.count(g, p, T.default_options(graph_capture=1))
    second, later = [], []
    for limit in range(40000, 40040):  # a wait limit that nothing reaches: another shape, the same launch
        o = T.default_options(graph_capture=1, wait_limit_ms=limit)
        for k in range(6):
            t0 = time.perf_counter()
            T.count(g, p, o)
            t = time.perf_counter() - t0
            if k:
                (second if k == 1 else later).append(t)
    # a capture takes several times as long as a replay of this launch
    assert statistics.median(second) < 2 * statistics.median(later)
