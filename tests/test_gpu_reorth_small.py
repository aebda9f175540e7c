"""Gram-Schmidt passes of the reorthogonalising mode on dimensions that give a
2048-row block to fewer than every SM (gs_small_kernel), needs a GB300.

Sizes: one row, below and above a warp, chunks per block 1, 2, 7, 8 (the change
from shared vectors to one chunk per warp), 9 and the last size before the
2048-row passes; Krylov dimensions around the groups of 16 vectors.

The mode's basis is orthogonal to rounding, so the run agrees with scipy's
exponential within tol (krylovTimeEvolver.cpp:153-254) plus rounding, and runs
with m vectors repeat bit for bit (integer sums).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(n, cplx):
    i = np.arange(n - 1)
    hop = np.full(n - 1, np.exp(0.3j) if cplx else 1.0 + 0j)
    d = np.arange(n)
    row, col = np.concatenate([i, i + 1, d]), np.concatenate([i + 1, i, d])
    val = np.concatenate([hop, np.conj(hop), np.cos(0.1 * d) + 0j])
    order = np.argsort(row * n + col, kind="stable")
    return row[order], col[order], val[order]


@pytest.mark.parametrize("n,m,cplx", [(1, 3, False), (5, 5, True), (33, 16, False), (700, 17, True), (4_900, 33, False),
                                      (9_000, 15, True), (34_020, 12, False), (38_700, 12, True), (43_100, 12, False),
                                      (311_000, 6, True)])
def test_reorth_small_dimensions(te_gpu, n, m, cplx):
    import scipy.sparse as sp
    from scipy.sparse.linalg import expm_multiply
    row, col, val = _chain(n, cplx)
    rng = np.random.default_rng(n)
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    v /= np.linalg.norm(v)
    M = te_gpu.Matrix(n, row, col, val)
    runs = []
    for _ in range(2):
        ev = te_gpu.Evolver(M, v, 0.5, 0.25, [], exp_factor=-1.3, tol=1e-9, m=m, reorth=True)
        runs.append(ev.time_evolve())
        ev.close()
    assert np.array_equal(runs[0]["state"], runs[1]["state"])
    exact = expm_multiply(1.3j * 0.5 * sp.csr_matrix((val, (row, col)), shape=(n, n)), v)
    assert np.linalg.norm(runs[0]["state"] - exact) < 1e-9 + 1e-12
