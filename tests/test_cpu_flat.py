"""The flat kernel's plan form (flat_plan.cpp), run in Python on small graphs
over every form the C ABI accepts -- symmetric and directed CSRs, self-loops,
labels -- and compared with the oracle's enumeration of the same plan.

The form: vertices 2..s are enumerated, each from the intersection of its
backward neighbours' rows under the conditions, or from the siblings of an
earlier level (reuse); the t vertices after s are counted from the sizes of
their candidate sets and of the sets' intersections."""
import random

import numpy as np
import pytest

from tests.golden.make_golden import random_pattern
from tests.patterns import CYCLE4, HOUSE, K4, K5, TRIANGLE, reference_patterns

NO_TERM = 255


def run_flat(rowptr, colidx, labels, plan, labeled):
    k, F = plan["k"], plan["flat"]
    n = len(rowptr) - 1
    N = [set(colidx[rowptr[v]:rowptr[v + 1]].tolist()) for v in range(n)]
    deg = np.diff(rowptr)
    maxnd = [max((int(deg[w]) for w in N[v]), default=-1) for v in range(n)]
    s, t = F["s"], F["t"]

    def cond(st, phi, x):
        _, label, larger, less, neq, _, _ = st
        if labeled and labels[x] != label:
            return False
        return all(not (larger >> j & 1 and x <= phi[j]) and not (less >> j & 1 and x >= phi[j])
                   and not (neq >> j & 1 and x == phi[j]) for j in range(len(phi)))

    def cands(st, phi, sets):
        c = set.intersection(*[N[phi[b]] for b in st[0]])
        out = {x for x in c if cond(st, phi, x)}
        if st[5]:  # the reuse level gives the same set
            r = set.intersection(sets[st[5]], *[N[phi[b]] for b in st[6]])
            assert {x for x in r if cond(st, phi, x)} == out
        return out

    def below(phi, sets):
        size = [0] * 8
        for m in range(1, 1 << t):
            if F["term_of"][m] != NO_TERM:
                size[m] = len(cands(F["terms"][F["term_of"][m]], phi, sets))
        a, b, c = size[1], size[2], size[4]
        if t == 1:
            return a
        if F["form"] == 1:
            return a * (a - 1) // 2 if t == 2 else a * (a - 1) * (a - 2) // 6
        if t == 2:
            return a * b - size[3]
        return a * b * c - size[3] * c - size[5] * b - size[6] * a + 2 * size[7]

    def rec(phi, sets):
        level = len(phi) - 1
        if level == s:
            return below(phi, sets)
        c = cands(F["steps"][level - 1], phi, sets)
        return sum(rec(phi + [x], {**sets, level + 1: c}) for x in c)

    total = 0
    want = plan["vertex_labels"]
    for r in range(n):
        for c in N[r]:
            if plan["orient"] and not labeled and not r < c:
                continue
            if labeled and (labels[r] != want[0] or labels[c] != want[1]):
                continue
            if deg[r] < plan["degree"][0] or deg[c] < plan["degree"][1] or maxnd[c] < plan["degree"][2]:
                continue
            total += rec([r, c], {})
    return total if labeled else total * plan["multiplicity"]


def graphs():
    """(name, rowptr, colidx) of small CSRs: symmetric, one-directional, with
    self-loops, and with a row that holds every vertex."""
    rng = random.Random(7)
    out = []
    for kind in ("symmetric", "directed", "loops", "hub"):
        n = 26
        e = set()
        while len(e) < 90:
            u, v = rng.randrange(n), rng.randrange(n)
            if u == v:
                continue
            e.add((u, v))
            if kind != "directed":
                e.add((v, u))
        if kind == "loops":
            e |= {(v, v) for v in range(0, n, 2)}
        if kind == "hub":
            e |= {(0, v) for v in range(1, n)} | {(v, 0) for v in range(1, n)}
        rows = [sorted(b for a, b in e if a == v) for v in range(n)]
        out.append((kind, np.array([0] + list(np.cumsum([len(r) for r in rows])), np.int64),
                    np.array([x for r in rows for x in r], np.int32)))
    return out


def texts():
    rng = random.Random(31)
    out = [TRIANGLE, CYCLE4, HOUSE, K4, K5] + [t for _, t in reference_patterns()]
    for edges in ("01 12 03 14 25", "01 12 02 03 13 14 24 25"):  # three independent last vertices
        out.append("".join(f"v {i} {i % 2}\n" for i in range(6)) +
                   "".join(f"e {e[0]} {e[1]} 1\n" for e in edges.split()))
    out += [random_pattern(3 + i % 4, 0.15 + 0.1 * (i % 6), 2, rng) for i in range(40)]
    return out


@pytest.mark.parametrize("labeled", [False, True])
def test_flat_form_equals_enumeration(T, po, labeled):
    seen = set()
    for kind, rowptr, colidx in graphs():
        labels = np.array([i * 7 % 3 % 2 for i in range(len(rowptr) - 1)], np.int32)
        ora = po.Graph(rowptr.copy(), colidx.copy(), labels.copy())
        for text in texts():
            plan = T.PatternPreprocessor(text=text, labeled=labeled).dump()
            if "flat" not in plan or plan["k"] > 6:
                continue
            want = po.count(ora, po.Plan(text, labeled))
            if want > (60000 if plan["flat"]["t"] == 1 else 3000000):
                continue  # too many nodes for Python
            assert run_flat(rowptr, colidx, labels, plan, labeled) == want, (kind, labeled, text)
            seen.add((plan["flat"]["t"], plan["flat"]["form"], any(st[5] for st in plan["flat"]["terms"])))
    # every way of counting was reached
    assert {(1, 0, False), (2, 0, False), (3, 0, False)} <= seen
    assert labeled or {(2, 1, False), (1, 0, True)} <= seen


def test_last_vertex_off_its_parent_needs_a_tail(T):
    """A plan whose last vertex does not hang on its parent has a flat form only
    when the tail counts it without enumerating its siblings."""
    for text in texts():
        for labeled in (False, True):
            plan = T.PatternPreprocessor(text=text, labeled=labeled).dump()
            if plan["k"] >= 4 and plan["k"] - 2 not in plan["backward_neighbors"][-1] and "flat" in plan:
                assert plan["flat"]["t"] >= 2
