"""Matrices from 2^14 entries in row order are laid out on the device; the same
entries with the rows out of order are converted on the host.  Each row keeps
its entries' order either way, so products are equal bit for bit."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("complex_values", [False, True])
@pytest.mark.parametrize("n,nnz", [(16383, 16383), (16384, 16384), (16385, 16384), (500, 16385), (3, 18000), (3000, 200001)])
def test_sorted_and_unsorted_rows(te_gpu, n, nnz, complex_values):
    rng = np.random.default_rng(n + nnz)
    row = np.sort(rng.integers(0, n, nnz))
    col = rng.integers(0, n, nnz)  # repeated entries add
    val = rng.standard_normal(nnz) + 1j * (rng.standard_normal(nnz) if complex_values else 0.0)
    moved = np.argsort(-row, kind="stable")  # rows last to first, each in its own order
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a, b = te_gpu.Matrix(n, row, col, val), te_gpu.Matrix(n, row[moved], col[moved], val[moved])
    assert np.array_equal(a.spmv(x), b.spmv(x))
    ia, ib = a.info(), b.info()
    assert {k: v for k, v in ia.items() if k != "norm1"} == {k: v for k, v in ib.items() if k != "norm1"}
    # column sums in another order: nnz roundings of a sum of nnz terms at most
    assert abs(ia["norm1"] - ib["norm1"]) <= nnz * np.finfo(float).eps * ia["norm1"]


def test_bad_entries_are_refused(te_gpu):
    n, nnz = 4000, 20000
    row, col = np.sort(np.arange(nnz) % n), np.arange(nnz) % n
    for r, c in ((n, 0), (0, n)):
        bad_row, bad_col = row.copy(), col.copy()
        bad_row[-1], bad_col[-1] = max(r, row[-1]), c or col[-1]
        with pytest.raises(Exception, match="out of range"):
            te_gpu.Matrix(n, bad_row, bad_col, np.ones(nnz, dtype=np.complex128))


@pytest.mark.parametrize("last", [False, True])
def test_a_long_row_stays_quick(te_gpu, last):
    """A long row among the sorted ones (an arrow matrix of 260 000 entries: the
    device would take a thread's time for each of its 86 666, 28 times the host's
    in all): the creation takes no longer than from rows out of order, which the
    host converts, but for what the rest of the creation varies (a factor 2)."""
    nnz = 260_000
    n = nnz // 3
    row = np.sort(np.r_[np.full(n, n - 1 if last else 0), np.arange(nnz - n) % n])
    col = np.arange(nnz) % n
    val = np.ones(nnz, dtype=np.complex128)
    moved = np.argsort(-row, kind="stable")

    def best(r, c):
        times = []
        for _ in range(6):
            start = time.perf_counter()
            te_gpu.Matrix(n, r, c, val).close()
            times.append(time.perf_counter() - start)
        return min(times)

    assert best(row, col) <= 2 * best(row[moved], col[moved])
