"""Schedule of batched evolutions: one instance, more than a warp of them, more
than the tile of the costs' prefix sums; running times that end instances early;
instances of a single chunk.

Each instance's occupations stay within the solver's error bound of the exact
ones: states within tol of each other differ by at most 2 N tol in an occupation
of at most N (plus the roundings, far below that).  The persistent launch builds
the same schedule: equal bit for bit."""
import numpy as np
import pytest

from oracle import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 31, 33, 200, 1025])
def test_batch_schedule(te_gpu, count):
    tol = 1e-9
    kinds = []
    for L in (2, 4, 5):
        states, H = models.bose_hubbard(L, L, 1.0, 2.0)
        n = len(states)
        dense = np.zeros((n, n))
        np.add.at(dense, (H[0], H[1]), H[2].real)
        diag = models.create_matrix([models.number_operator(0, 1.0)], states)
        n0 = np.zeros(n)
        np.add.at(n0, diag[0], diag[2].real)
        v = np.zeros(n, dtype=np.complex128)
        v[models.index_of(states, [L] + [0] * (L - 1))] = 1.0
        kinds.append((L, te_gpu.Matrix.from_coo(n, H), te_gpu.Matrix.from_coo(n, diag), v, n0, *np.linalg.eigh(dense)))
    rng = np.random.default_rng(count)
    picks = rng.integers(0, len(kinds), count)
    times = rng.choice([0.5, 1.0, 4.0], count)
    inst = [dict(H=kinds[k][1], v=kinds[k][3], t=float(t), sampling_step=float(t) / 4, tol=tol, m=12,
                 observables=[kinds[k][2]]) for k, t in zip(picks, times)]
    samples = []
    for persistent in (False, True):
        batch = te_gpu.Batch(inst, persistent=persistent)
        batch.run()
        samples.append([batch.samples(i) for i in range(count)])
    for i, (k, t) in enumerate(zip(picks, times)):
        assert np.array_equal(samples[0][i], samples[1][i]), i
        L, _, _, v, n0, e, q = kinds[k]
        ts = t / 4 * np.arange(5)
        psi = q @ (np.exp(-1j * np.outer(e, ts)) * (q.conj().T @ v)[:, None])
        assert np.max(np.abs(np.ravel(samples[0][i]) - n0 @ np.abs(psi) ** 2)) <= 2 * L * tol, i
