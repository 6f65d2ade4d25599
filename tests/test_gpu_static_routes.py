"""tdfs_count_static takes the flat kernel where the plan has its form and the row
tables fit the fixed array beside the other parts, else the DFS kernel: both
give tdfs_count's counts, in any order of calls on the one array, and refuse
the same labels."""
import random
import re

import numpy as np
import pytest

from tests.golden.make_golden import random_pattern
from tests.patterns import CYCLE4, HOUSE, TRIANGLE, clique

FORMAT = 2
KERNELS = [{}, {"tail_count": 1}, {"merge_window": 128}, {"steal": 0}]  # flat, then DFS by three knobs


def on_device(csr):
    import torch
    out = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (csr.rowptr, csr.colidx)]
    out.append(None if csr.labels is None else torch.from_numpy(np.ascontiguousarray(csr.labels)).cuda())
    torch.cuda.synchronize()
    return out


def static(T, csr, dev, P, **kw):
    return T.count_static(0, csr.n, csr.nedges, dev[0].data_ptr(), dev[1].data_ptr(),
                          None if dev[2] is None else dev[2].data_ptr(), P, T.default_options(**kw))


@pytest.mark.gpu
def test_calls_of_either_kernel_follow_one_another(T):
    rng = random.Random(17)
    graphs = [T.gen_er(4096, 16.0, 0).set_labels(4, 2), T.gen_er(1001, 7.0, 3).set_labels(20, 1),
              T.gen_chung_lu(20000, 60000, 2.1, 600, 1).set_labels(4, 2)]
    assert any(g.nedges % 4 for g in graphs)
    for csr in graphs:
        G, dev = T.GraphPreprocessor(csr=csr, labeled=True), on_device(csr)
        texts = [(TRIANGLE, False), (CYCLE4, False), (HOUSE, False), (clique(4), False)]
        texts += [(random_pattern(3 + i, 0.5, 4, rng), True) for i in range(4)]
        jobs = [(T.PatternPreprocessor(text=t, labeled=lab), kw) for t, lab in texts for kw in KERNELS]
        want = {id(P): T.count(G, P).count for P, _ in jobs}
        rng.shuffle(jobs)
        for P, kw in jobs + jobs[::-1]:
            assert static(T, csr, dev, P, **kw) == want[id(P)], (P.dump(), kw)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", KERNELS[:2])
@pytest.mark.parametrize("bad", [-1, 255, 1 << 20])
def test_labels_out_of_range_are_refused(T, kw, bad):
    csr = T.gen_er(2000, 10.0, 1).set_labels(3, 1)
    P = T.PatternPreprocessor(text="v 0 1\nv 1 0\nv 2 2\ne 0 1 1\ne 0 2 1\ne 1 2 1\n", labeled=True)
    dev = on_device(csr)
    want = static(T, csr, dev, P, **kw)
    dev[2][1999] = bad
    with pytest.raises(T.TdfsError) as e:
        static(T, csr, dev, P, **kw)
    assert e.value.code == FORMAT and "[0, 254]" in str(e.value)
    dev[2][1999] = int(csr.labels[1999])
    assert static(T, csr, dev, P, **kw) == want == T.count(T.GraphPreprocessor(csr=csr, labeled=True), P).count


def first_edges(T, csr, pairs):
    """The CSR of the first so many vertex pairs of a symmetric one."""
    src = np.repeat(np.arange(csr.n), np.diff(csr.rowptr))
    keep = np.flatnonzero(src < csr.colidx)[:pairs]
    u, v = src[keep], csr.colidx[keep].astype(np.int64)
    both = np.sort(np.concatenate([u * csr.n + v, v * csr.n + u]))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(both // csr.n, minlength=csr.n))])
    return T.csr_from_arrays(rowptr, both % csr.n)


@pytest.mark.gpu
def test_where_the_tables_stop_fitting(T):
    """The largest graph whose tables fit the array, and the next larger ones."""
    n, E = 60000, 8_000_000
    P = [T.PatternPreprocessor(text=t) for t in (TRIANGLE, clique(4))]
    with pytest.raises(T.TdfsError) as e:  # refused from the sizes alone: what the parts but the tables take
        T.count_static(0, n, E, 256, 256, None, P[0])
    need, have = (int(re.search(t, str(e.value)).group(1)) for t in (r"needs (\d+) bytes", r"holds (\d+) bytes"))
    line = (have - (need - 4 * E) - 32 * n) // 14  # 4 bytes per edge for its source, 10 for its table
    full = T.gen_er(n, 36.0, 5)
    assert full.nedges > line + 100_000
    for pairs in (line // 2 - 50, line // 2 - 1, line // 2, line // 2 + 1, line // 2 + 50, line // 2 + 20_000):
        csr = first_edges(T, full, pairs)
        assert csr.nedges == 2 * pairs
        G, dev = T.GraphPreprocessor(csr=csr), on_device(csr)
        for p in P:
            assert static(T, csr, dev, p) == T.count(G, p).count, pairs
        G.close()
