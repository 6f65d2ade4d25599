"""The workloads whose speed is tracked, as a program that uses this package runs them.

A case names a graph recipe, the patterns counted on it and the entry point the
program calls.  Graphs are made here from the seed alone (host CSR arrays, as a
loader leaves them): `er` Erdos-Renyi, `cl` Chung-Lu power law with ids in
descending degree, `rmat` R-MAT, deduplicated and symmetrised.  Patterns are
names from NAMED or "labels:edges" codes ("3211:01,02,12,13,23" is four
vertices labeled 3, 2, 1, 1); a case with labels > 0 counts them labeled.
"""
import math
import random

import numpy as np
import torch

import tdfs_b200 as T

NAMED = {
    "triangle": "111:01,02,12",
    "cycle4": "1111:01,12,23,03",
    "diamond": "1111:01,02,03,12,13",
    "clique4": "1111:01,02,03,12,13,23",
    "clique5": "11111:01,02,03,04,12,13,14,23,24,34",
    "clique6": "111111:01,02,03,04,05,12,13,14,15,23,24,25,34,35,45",
    "house": "11111:01,02,12,13,24,34",
}

SMALL = "triangle cycle4 diamond clique4"
# eight random connected 6-7 vertex patterns, density 0.4, labels in [0, 4)
TREES = ("201033:01,05,12,13,24 0022032:01,04,06,12,15,23,24,35 321221:01,05,12,23,24 "
         "1012222:01,02,03,04,12,13,25,35,46,56 131223:01,05,12,14,23,45 2001011:01,12,14,15,23,36 "
         "020120:01,12,23,34,45 0111000:01,03,04,06,12,24,25,45")
# random connected 4-6 vertex patterns, density 0.45, labels in [0, 4)
MIXED = ("3211:01,02,12,13,23 02023:01,03,04,12,13,14,23,24,34 3333:01,02,03,12,13 03102:01,03,04,12,23,24 "
         "300121:01,03,04,12,13,23,24,25,34,45 3103:01,02,03,12,13,23 30030:01,12,13,14,23,24,34")


def listed():
    return [
        # a single small query: nothing but latency and launches
        dict(name="er_triangle", entry="count", graph="er", n=4096, degree=16, labels=0, patterns="triangle"),
        # the small unlabeled set, one replayed batched launch
        dict(name="er_unlabeled_batch", entry="batch", graph="er", n=4096, degree=16, labels=0, patterns=SMALL,
             captured=True),
        # the small labeled set of uneven 6-7 vertex patterns, one replayed batched launch
        dict(name="er_labeled_batch", entry="batch", graph="er", n=4096, degree=16, labels=4, patterns=TREES,
             captured=True),
        # a whole request from host arrays: upload, compile, count both modes, free
        dict(name="er_whole_step", entry="step", graph="er", n=4096, degree=16, labels=4,
             patterns=SMALL + " " + TREES, captured=True),
        # a caller that owns the device memory: no allocation, everything derived per call; ragged size
        dict(name="er_static_cycle4", entry="static", graph="er", n=20011, degree=11, labels=0, patterns="cycle4"),
        # a burst of 64 random labeled 3-7 vertex queries in one launch
        dict(name="er_query_burst", entry="batch", graph="er", n=4096, degree=16, labels=4, patterns="random",
             pattern_seed=5, queries=64, captured=False),
        # power law, hubs far above the buffers, default options
        dict(name="cl_unlabeled_batch", entry="batch", graph="cl", n=50000, degree=6, cap=3000, labels=0,
             patterns="triangle cycle4 clique4 clique5", captured=False),
        # power law, random labeled queries of uneven size in one launch
        dict(name="cl_labeled_batch", entry="batch", graph="cl", n=50000, degree=6, cap=3000, labels=4,
             patterns=MIXED, captured=False),
        # loading a large labeled graph from host arrays and asking one cheap question
        dict(name="cl_load_and_count", entry="step", graph="cl", n=1100000, degree=5.4545, cap=30000, labels=4,
             patterns="012:01,02,12", captured=False),
        # 5-cliques of the large power-law graph: one rank's share of an 8-rank job
        dict(name="cl_clique5_rank", entry="count", graph="cl", n=1100000, degree=5.4545, cap=30000, labels=0,
             patterns="clique5", ranks=8, rank=3),
        # houses of the large power-law graph over a slice of its edges
        dict(name="cl_house_slice", entry="count", graph="cl", n=1100000, degree=5.4545, cap=30000, labels=0,
             patterns="house", begin=0.5, share=1 / 2000),
        # 4-cliques of a skewed R-MAT graph: one rank's share of an 8-rank job
        dict(name="rmat_clique4_rank", entry="count", graph="rmat", scale=18, degree=16, labels=0,
             patterns="clique4", ranks=8, rank=6),
    ]


def random_pattern(rng, k, density, labels):
    """Connected, every vertex with an earlier neighbour, 2 next to 1."""
    edges = {(1 if i == 2 else rng.randrange(i), i) for i in range(1, k)}
    edges |= {(i, j) for i in range(k) for j in range(i + 1, k) if rng.random() < density}
    return "".join(str(rng.randrange(labels)) for _ in range(k)) + ":" + ",".join("%d%d" % e for e in sorted(edges))


def log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("er_count", "er_batch", "er_labeled", "er_step", "er_static", "er_burst", "cl_batch",
                       "cl_labeled", "cl_load", "cl_clique", "cl_house", "rmat"))
    if kind.startswith("er_"):
        c = dict(graph="er", n=int(log_uniform(rng, 1000, 24000)), degree=rng.randint(8, 20), labels=0)
        if kind == "er_count":
            c.update(entry="count", patterns=rng.choice(("triangle", "cycle4", "diamond", "house")))
        elif kind == "er_batch":
            c.update(entry="batch", patterns=" ".join(["cycle4"] + rng.sample(sorted(set(NAMED) - {"cycle4"}), 3)),
                     captured=rng.random() < 0.5)
        elif kind == "er_static":
            c.update(entry="static", patterns=rng.choice(("triangle", "cycle4", "diamond", "house")))
        else:
            c.update(n=int(log_uniform(rng, 1000, 8000)), degree=rng.randint(8, 16), labels=4)
            queries = [random_pattern(rng, rng.randint(5, 7), rng.uniform(0.05, 0.3), 4) for _ in range(6)]
            if kind == "er_labeled":
                c.update(entry="batch", patterns=" ".join(queries), captured=rng.random() < 0.5)
            elif kind == "er_step":
                c.update(entry="step", patterns=" ".join(["triangle", "diamond"] + queries),
                         captured=rng.random() < 0.5)
            else:
                c.update(entry="batch", patterns="random", pattern_seed=rng.randrange(1 << 20),
                         queries=int(log_uniform(rng, 8, 128)), captured=rng.random() < 0.5)
    elif kind == "rmat":
        c = dict(graph="rmat", scale=rng.randint(13, 18), degree=rng.randint(8, 16), labels=0, entry="count",
                 patterns=rng.choice(("clique4", "triangle")), ranks=rng.randint(8, 32), rank=rng.randrange(8))
    else:
        n = int(log_uniform(rng, 20000, 60000 if kind in ("cl_batch", "cl_labeled") else 1100000))
        c = dict(graph="cl", n=n, degree=round(rng.uniform(4, 6), 3), cap=int(min(30000, n / 20)), labels=0)
        if kind == "cl_batch":
            c.update(entry="batch", patterns=" ".join(rng.sample(("triangle", "diamond", "clique4", "clique5"), 3)),
                     captured=rng.random() < 0.5)
        elif kind == "cl_labeled":
            c.update(entry="batch", labels=4, captured=rng.random() < 0.5,
                     patterns=" ".join(random_pattern(rng, rng.randint(3, 5), rng.uniform(0.5, 0.8), 4)
                                       for _ in range(4)))
        elif kind == "cl_load":
            c.update(entry="step", labels=rng.randint(3, 8), patterns="012:01,02,12", captured=False)
        elif kind == "cl_clique":
            c.update(entry="count", patterns=rng.choice(("triangle", "clique4", "clique5")), ranks=rng.randint(10, 32),
                     rank=rng.randrange(8))
        else:
            c.update(entry="count", patterns="house", begin=rng.uniform(0.5, 0.9),
                     share=log_uniform(rng, 1 / 16000, 1 / 3000))
    return c


# ---- inputs -------------------------------------------------------------------

def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def distinct_pairs(propose, n, want):
    """`want` distinct unordered pairs u < v from a proposal distribution."""
    keys = torch.empty(0, dtype=torch.int64, device=device())
    for _ in range(16):
        u, v = propose(max(1024, int(1.3 * (want - len(keys)))))
        lo, hi = torch.minimum(u, v), torch.maximum(u, v)
        keys = torch.unique(torch.cat([keys, (lo * n + hi)[lo < hi]]))
        if len(keys) >= want:
            break
    return keys


def graph_arrays(case, seed):
    """(rowptr int64, colidx int32, labels int32 or None) on the device."""
    g = torch.Generator(device=device()).manual_seed(seed)
    rand = lambda m: torch.rand(m, generator=g, device=device(), dtype=torch.float64)  # noqa: E731
    n = case.get("n") or 1 << case["scale"]
    want = int(n * case["degree"] / 2)
    if case["graph"] == "er":
        keys = distinct_pairs(lambda m: ((rand(m) * n).long(), (rand(m) * n).long()), n, want)
    elif case["graph"] == "cl":
        # expected degrees ~ i^(-1/(gamma-1)), gamma 2.1, the largest capped
        w = np.arange(1, n + 1, dtype=np.float64) ** (-1 / 1.1)
        w = np.minimum(w * (2 * want / w.sum()), case["cap"])
        cum = torch.from_numpy(np.cumsum(w) / w.sum()).to(device())
        ends = lambda m: torch.searchsorted(cum, rand(m)).clamp_(max=n - 1)  # noqa: E731
        keys = distinct_pairs(lambda m: (ends(m), ends(m)), n, want)
    else:  # quadrants 0.57, 0.19, 0.19, 0.05 per bit
        u = torch.zeros(int(n * case["degree"]), dtype=torch.int64, device=device())
        v = torch.zeros_like(u)
        for _ in range(case["scale"]):
            r = rand(len(u))
            u = 2 * u + (r >= 0.76)
            v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        lo, hi = torch.minimum(u, v), torch.maximum(u, v)
        keys = torch.unique((lo * n + hi)[lo < hi])
        want = len(keys)
    keys = keys[torch.randperm(len(keys), generator=g, device=device())[:want]]
    lo, hi = keys // n, keys % n
    if case["graph"] == "cl":
        deg = torch.bincount(torch.cat([lo, hi]), minlength=n)
        rank = torch.empty(n, dtype=torch.int64, device=device())
        rank[torch.argsort(deg, descending=True, stable=True)] = torch.arange(n, device=device())
        lo, hi = rank[lo], rank[hi]
    both = torch.sort(torch.cat([lo * n + hi, hi * n + lo])).values
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=device())
    rowptr[1:] = torch.cumsum(torch.bincount(both // n, minlength=n), 0)
    labels = (rand(n) * case["labels"]).int() if case["labels"] else None
    return rowptr, (both % n).int(), labels


def pattern_codes(case):
    if case["patterns"] == "random":
        rng = random.Random(case["pattern_seed"])
        return [random_pattern(rng, rng.randint(3, 7), rng.uniform(0.1, 0.6), case["labels"])
                for _ in range(case["queries"])]
    return case["patterns"].split()


def pattern_list(case):
    """[(text in the .g format, labeled)]: named patterns are counted unlabeled."""
    out = []
    for code in pattern_codes(case):
        labels, edges = NAMED.get(code, code).split(":")
        text = "# pattern\n" + "".join("v %d %s\n" % (i, c) for i, c in enumerate(labels))
        text += "".join("e %s %s 1\n" % (e[0], e[1]) for e in edges.split(","))
        out.append((text, code not in NAMED))
    return out


def prepare(case, seed):
    rowptr, colidx, labels = graph_arrays(case, seed)
    s = dict(case=case, texts=pattern_list(case))
    kw = dict(graph_capture=1) if case.get("captured") else {}
    if "share" in case:
        e = len(colidx)
        kw.update(edge_begin=int(case["begin"] * e), edge_end=int((case["begin"] + case["share"]) * e) + 1)
    if "ranks" in case:
        s["options"] = T.shard_options(case["rank"], case["ranks"], **kw)
    else:
        s["options"] = T.default_options(**kw) if kw else None
    if case["entry"] == "static":
        s.update(rowptr=rowptr, colidx=colidx)
    else:
        s.update(rowptr=rowptr.cpu().numpy(), colidx=colidx.cpu().numpy(),
                 labels=None if labels is None else labels.cpu().numpy())
    if case["entry"] not in ("step", "static"):
        s["graph"] = T.GraphPreprocessor(rowptr=s["rowptr"], colidx=s["colidx"], labels=s["labels"],
                                         labeled=labels is not None)
    if case["entry"] != "step":
        s["plans"] = [T.PatternPreprocessor(text=t, labeled=lab) for t, lab in s["texts"]]
    return s


def run(s):
    entry = s["case"]["entry"]
    if entry == "count":
        return T.count(s["graph"], s["plans"][0], s["options"]).count
    if entry == "batch":
        return np.array(T.count_batch(s["graph"], s["plans"], s["options"])[0], dtype=np.int64)
    if entry == "static":
        return T.count_static(0, len(s["rowptr"]) - 1, len(s["colidx"]), s["rowptr"].data_ptr(),
                              s["colidx"].data_ptr(), None, s["plans"][0])
    graph = T.GraphPreprocessor(rowptr=s["rowptr"], colidx=s["colidx"], labels=s["labels"], labeled=True)
    plans = [T.PatternPreprocessor(text=t, labeled=lab) for t, lab in s["texts"]]
    counts = T.count_batch(graph, plans, s["options"])[0]
    graph.close()
    return np.array(counts, dtype=np.int64)


def work(case):
    """The graph read once and one count written per pattern."""
    n = case.get("n") or 1 << case["scale"]
    edges = n * case["degree"] * (2 if case["graph"] == "rmat" else 1)
    return {"bytes": 8 * (n + 1) + 4 * edges + (4 * n if case["labels"] else 0) + 8 * len(pattern_codes(case)),
            "flops": 0}


# ---- the counts, restated -----------------------------------------------------

def embeddings(rowptr, colidx, labels, text, labeled):
    """Injective edge-preserving maps of one pattern, level by level over all
    partial maps of a block of first edges at a time."""
    lines = [x.split() for x in text.splitlines()]
    want = [int(x[2]) for x in lines if x[0] == "v"]
    adj = {frozenset((int(x[1]), int(x[2]))) for x in lines if x[0] == "e"}
    k, n = len(want), len(rowptr) - 1
    deg = rowptr[1:] - rowptr[:-1]
    src = torch.repeat_interleave(torch.arange(n, device=rowptr.device), deg)
    keys = src * n + colidx
    fits = lambda v, i: (labels[v] == want[i]) if labeled else torch.ones_like(v, dtype=torch.bool)  # noqa: E731
    total = 0
    for b in range(0, len(colidx), 4096):
        maps = torch.stack([src[b:b + 4096], colidx[b:b + 4096].long()], 1)
        maps = maps[fits(maps[:, 0], 0) & fits(maps[:, 1], 1) & (maps[:, 0] != maps[:, 1])]
        for i in range(2, k):
            back = [j for j in range(i) if frozenset((j, i)) in adj]
            d = deg[maps[:, back[0]]]
            row = torch.repeat_interleave(torch.arange(len(maps), device=d.device), d)
            at = torch.arange(len(row), device=d.device) - torch.repeat_interleave(torch.cumsum(d, 0) - d, d)
            x = colidx[rowptr[maps[row, back[0]]] + at].long()
            ok = fits(x, i)
            for j in range(i):
                ok &= maps[row, j] != x
            row, x = row[ok], x[ok]
            for j in back[1:]:
                key = maps[row, j] * n + x
                hit = keys[torch.searchsorted(keys, key).clamp_(max=len(keys) - 1)] == key
                row, x = row[hit], x[hit]
            if i == k - 1:
                total += len(x)
            else:
                maps = torch.cat([maps[row], x[:, None]], 1)
    return total


def exact(case, seed):
    # enumerating every map level by level is quick on the sparse graphs only, and
    # for patterns that many labels or few vertices keep small
    if case["graph"] != "er" or case["n"] > 5000 or "random" in case["patterns"] or "house" in case["patterns"]:
        return None
    arrays = graph_arrays(case, seed)
    counts = [embeddings(*arrays, text, labeled) for text, labeled in pattern_list(case)]
    return counts[0] if case["entry"] in ("count", "static") else np.array(counts, dtype=np.int64)
