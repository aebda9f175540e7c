"""Observables of whole sample batches (needs a GB300): diagonal, vector, general
sparse and dense observables against the same expectation values computed on
the host from the sampled states (callback observables, one sample at a time).

Sizes: below a warp, around a block, the row blocks that get a block per sample
and those that loop over the samples (above 64 blocks), more than 8 diagonal
and 2 vector observables (several launches), more than 16 samples per step
(several batches); observables with empty rows.

Both runs evolve the same state bit for bit (observables do not feed back), so
a value differs by the rounding of its sum only: at most n terms of O(1) total
in different orders, below 1e-12 of ||O||.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(n, seed, cplx):
    rng = np.random.default_rng(seed)
    i = np.arange(n - 1)
    hop = rng.uniform(0.5, 1.0, n - 1) * (np.exp(0.7j) if cplx else 1.0)
    row, col = np.concatenate([i, i + 1]), np.concatenate([i + 1, i])
    val = np.concatenate([hop, np.conj(hop)]).astype(np.complex128)
    order = np.argsort(row * n + col, kind="stable")
    return row[order], col[order], val[order]


@pytest.mark.parametrize("n,n_diag,n_vec,dense", [(20, 1, 0, True), (257, 9, 3, True), (1700, 8, 1, False),
                                                  (16_400, 3, 2, False), (40_001, 2, 0, False)])
def test_batched_observables_equal_host_values(te_gpu, n, n_diag, n_vec, dense):
    rng = np.random.default_rng(n)
    H = te_gpu.Matrix.from_coo(n, _chain(n, 1, False))
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    v /= np.linalg.norm(v)
    obs, host = [], []
    for k in range(n_diag):
        d = rng.uniform(-1.0, 1.0, n)
        d[k % n] = 0.0
        keep = np.nonzero(d)[0]
        obs.append(("sparse", te_gpu.Matrix.from_coo(n, (keep, keep, d[keep].astype(np.complex128)))))
        host.append(lambda x, d=d: float(np.sum(d * np.abs(x) ** 2)))
    for cplx in (False, True):
        r, c, w = _chain(n, 5 + cplx, cplx)
        keep = (r % 7 != 3) & (c % 7 != 3)  # empty rows
        r, c, w = r[keep], c[keep], w[keep]
        obs.append(("sparse", te_gpu.Matrix.from_coo(n, (r, c, w))))
        host.append(lambda x, r=r, c=c, w=w: float(np.sum(np.conj(x[r]) * w * x[c]).real))
    for k in range(n_vec):
        o = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        o /= np.linalg.norm(o)
        obs.append(("vector", o))
        host.append(lambda x, o=o: float(np.abs(np.vdot(x, o)) ** 2))
    if dense:
        A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        D = (A + A.conj().T) / (4 * np.sqrt(n))
        obs.append(("dense", D))
        host.append(lambda x, D=D: float(np.vdot(x, D @ x).real))
    a = te_gpu.Evolver(H, v, 2.0, 0.05, obs, tol=1e-9, m=20)
    b = te_gpu.Evolver(H, v, 2.0, 0.05, [("callback", f) for f in host], tol=1e-9, m=20)
    ra, rb = a.time_evolve(), b.time_evolve()
    a.close()
    b.close()
    assert ra["num_samples"] == rb["num_samples"] == 41
    assert np.array_equal(ra["state"], rb["state"])
    assert np.max(np.abs(ra["samples"] - rb["samples"])) < 2e-12
    assert np.min(np.max(np.abs(ra["samples"]), axis=1)) > 0.0
