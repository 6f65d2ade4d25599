"""What is wrong with a malformed CSR: the fault in the lowest row is the one
reported, however many there are and whichever thread finds which, and nothing
is read outside the arrays."""
import numpy as np
import pytest

from tests.test_gpu_flat import edge_graph


def message(make, rowptr, colidx):
    with pytest.raises(Exception) as e:
        make(rowptr, colidx)
    assert e.value.code == 2
    return str(e.value)


def broken(rowptr, colidx):
    """(rowptr, colidx, what the message says): one to three faults each."""
    n, E = len(rowptr) - 1, len(colidx)
    rows = [v for v in range(n) if rowptr[v + 1] - rowptr[v] >= 2]
    a, b, c = rows[3], rows[len(rows) // 2], rows[-2]

    def edit(*faults):
        r, x = rowptr.copy(), colidx.copy()
        for kind, v in faults:
            if kind == "range":
                x[r[v]] = n
            elif kind == "negative":
                x[r[v]] = -1
            elif kind == "order":
                x[r[v] + 1] = x[r[v]]
            elif kind == "falls":
                r[v + 1] = r[v] - 1
            elif kind == "beyond":
                r[v + 1] = E + 5
            elif kind == "below":
                r[v + 1] = -7
        return r, x

    says = {"range": "neighbour id out of range in row %d", "negative": "neighbour id out of range in row %d",
            "order": "row %d not strictly", "falls": "rowptr decreases at vertex %d",
            "beyond": "rowptr decreases at vertex %d", "below": "rowptr decreases at vertex %d"}
    for k1 in says:
        yield (*edit((k1, b)), says[k1] % b)
        for k2 in says:
            yield (*edit((k2, c), (k1, a)), says[k1] % a)
            yield (*edit((k2, c), (k1, a), (k2, b)), says[k1] % a)


def test_the_lowest_fault_is_reported(T):
    rowptr, colidx = edge_graph()
    T.csr_from_arrays(rowptr, colidx)
    for r, x, want in broken(rowptr, colidx):
        assert want in message(T.csr_from_arrays, r, x)


def test_the_lowest_fault_is_reported_by_many_threads(T):
    n, d = 300_000, 8  # enough for the check to be split over threads
    colidx = np.tile(np.arange(d, dtype=np.int32), n)
    rowptr = np.arange(n + 1, dtype=np.int64) * d
    for first in (5, n // 2, n - 300):
        x = colidx.copy()
        for v in list(range(first, n, 50)):
            x[v * d + 3] = -1 if v % 100 else 9
        want = "row %d" % first
        for _ in range(5):
            assert want + " " in message(T.csr_from_arrays, rowptr, x) + " "


@pytest.mark.gpu
def test_the_device_check_says_what_the_host_says(T):
    rowptr, colidx = edge_graph()
    make = lambda r, x: T.GraphPreprocessor(rowptr=r, colidx=x)  # noqa: E731
    make(rowptr, colidx)
    for r, x, want in broken(rowptr, colidx):
        got = message(make, r, x)
        assert want in got and got == message(T.csr_from_arrays, r, x)
