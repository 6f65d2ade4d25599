"""Work stealing in the DFS kernel never counts an item twice.

A hoisted level's core set (the candidates that depend on an earlier level
only) is built once and published per node.  Items a thief can see must be
published exactly once: a plan with such a level, split as eagerly as the
options allow on a graph with hubs, is counted many times over and equals the
enumeration on the CPU every time."""
import pytest

pytestmark = pytest.mark.gpu

# vertex 3 hangs on 0 and 1 only (its set is shared by all of vertex 2's candidates)
LABELED = ("v 0 1\nv 1 0\nv 2 0\nv 3 1\nv 4 0\nv 5 1\ne 0 1 1\ne 0 2 1\ne 0 3 1\ne 0 4 1\ne 1 2 1\ne 1 3 1\ne 1 4 1\n"
           "e 1 5 1\ne 2 4 1\ne 2 5 1\ne 3 4 1\ne 3 5 1\ne 4 5 1\n")
UNLABELED = "v 0 1\nv 1 1\nv 2 1\nv 3 1\nv 4 1\ne 0 1 1\ne 0 2 1\ne 1 2 1\ne 1 3 1\ne 2 4 1\ne 3 4 1\n"


@pytest.mark.parametrize("text,labeled", [(LABELED, True), (UNLABELED, False)])
@pytest.mark.parametrize("opt", [{}, {"work_budget": 10 ** 12}, {"label_rows": -1}])
def test_hoisted_levels_under_eager_splitting(T, po, text, labeled, opt):
    csr = T.gen_chung_lu(20000, 60000, 2.1, 600, 1).set_labels(2, 2)
    P = T.PatternPreprocessor(text=text, labeled=labeled)
    if not labeled:  # a slice that holds many of the matches
        opt = dict(opt, edge_begin=csr.nedges // 2, edge_end=csr.nedges // 2 + csr.nedges // 50)
    G = T.GraphPreprocessor(csr=csr, labeled=True)
    want = T.count(G, P, T.default_options(**{k: v for k, v in opt.items() if k.startswith("edge_")})).count
    if labeled:
        assert want == po.count(po.Graph(csr.rowptr.copy(), csr.colidx.copy(), csr.labels.copy()), po.Plan(text, True))
    o = T.default_options(split_after_us=-1, tail_count=1, **opt)  # (tail_count: the DFS kernel)
    got = [T.count(G, P, o).count for _ in range(60)]
    assert want > 0 and set(got) == {want}
