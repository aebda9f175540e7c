"""The one-launch Lanczos kernels (te_step.cu below 2048 chunks of 32 rows,
te_resident.cu from there on) against the per-iteration passes
(TE_OPT_FUSED_LANCZOS 0); needs a GB300.

Sizes sit at the edges of the kernels' layouts: one row, one chunk, chunks per
warp 1 / 2 / more than 4 (rows re-read), one and several groups of 32 blocks,
more blocks than SMs, slots beyond shared memory, the change from one kernel
to the other, chunks per warp 1..4 of the resident kernel, its last size, and
rows streamed beyond it (limbs, dictionary, complex).

Both runs are within tol of the exact state (krylovTimeEvolver.cpp:153-254),
so their states agree within 2 tol; with a random start vector (no Ritz value
converges within the Krylov dimension) the coefficients agree to rounding, so
the steps are the same and their sizes agree to 1e-9 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-9


def _matrix(te, n, per_row, seed, cplx, hub=0, values=None):
    """Random Hermitian matrix of about 2 per_row entries per row, norm about 1;
    hub: so many entries in row 0 (and column 0)."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), per_row)
    c = rng.integers(0, n, size=len(r))
    if hub:
        r = np.concatenate([r, np.zeros(hub, dtype=np.int64)])
        c = np.concatenate([c, rng.integers(0, n, size=hub)])
    v = rng.standard_normal(len(r)) + (1j * rng.standard_normal(len(r)) if cplx else 0.0)
    if values:
        v = np.array(values)[rng.integers(0, len(values), size=len(r))] + 0j
    v = v / (4.0 * np.sqrt(per_row + hub))
    row, col, val = np.concatenate([r, c]), np.concatenate([c, r]), np.concatenate([v, np.conj(v)])
    order = np.argsort(row * n + col, kind="stable")
    return te.Matrix(n, row[order], col[order], val[order])


def _run(te, M, v, fused, fixed, exp_factor):
    ev = te.Evolver(M, v, 12.0, 3.0, [("vector", v)], exp_factor=exp_factor, tol=TOL, m=24)
    ev.set_option(te.OPT_FUSED_LANCZOS, fused)
    ev.set_option(te.OPT_FIXED_SPMV, fixed)
    out = ev.time_evolve(trace=True)
    ev.close()
    return out


CASES = [
    # n, per_row, complex, hub, few values, launches of the Lanczos iterations in one
    (1, 1, False, 0, None), (31, 3, True, 0, None), (32, 3, False, 0, None), (33, 2, False, 0, None),
    (257, 4, True, 0, None), (900, 2, False, 700, None), (8192, 6, False, 0, (1.0, -0.5)),
    (8225, 5, True, 0, None), (3000, 300, False, 0, None), (39_000, 4, False, 0, None), (48_001, 3, True, 0, None),
    (65_504, 3, False, 0, None), (65_536, 3, False, 0, (0.5, 1.0, 2.0)), (70_001, 4, True, 0, None),
    (100_000, 3, False, 0, None), (185_000, 2, False, 0, (1.0, -1.0)), (280_003, 2, True, 0, None),
    (369_664, 2, False, 0, None), (369_665, 2, False, 0, None), (400_001, 2, True, 0, None),
    (900_000, 2, False, 0, (1.0, -0.5)), (1_000_003, 3, True, 0, None),
]


@pytest.mark.parametrize("n,per_row,cplx,hub,values", CASES)
def test_one_launch_equals_passes(te_gpu, n, per_row, cplx, hub, values):
    M = _matrix(te_gpu, n, per_row, n + per_row, cplx, hub, values)
    rng = np.random.default_rng(3)
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    v /= np.linalg.norm(v)
    for fixed, exp_factor in ((1, 1.0), (0, -0.7)):
        a, b = _run(te_gpu, M, v, 1, fixed, exp_factor), _run(te_gpu, M, v, 0, fixed, exp_factor)
        assert a["n_steps"] == b["n_steps"] and a["status"] == b["status"]
        assert a["num_samples"] == b["num_samples"] and a["krylov_dim"] == b["krylov_dim"]
        assert np.linalg.norm(a["state"] - b["state"]) < 2 * TOL
        assert np.max(np.abs(a["samples"] - b["samples"])) < 4 * TOL
        for x, y in zip(a["trace"], b["trace"]):
            assert x["breakdown"] == y["breakdown"] and x["m_eff"] == y["m_eff"]
            assert abs(x["t_step"] - y["t_step"]) <= 1e-9 * y["t_step"]
        # the passes take 2 launches per iteration, the one-launch kernels 1 per step
        steps = a["n_steps"]
        if n >= 24 and (fixed or n <= 369_664):
            assert b["launches"] - a["launches"] == (2 * 24 - 1) * steps
        elif n > 369_664:  # the rows are streamed on the fixed-point path only
            assert b["launches"] == a["launches"]


def test_resident_exchange_timeout(te_gpu):
    """A wait of the resident kernel that runs out (every exchange waits for one
    block more than the grid has): TE_ERR_DEVICE_TIMEOUT, and the same evolver
    then runs to the passes' result."""
    n = 70_000
    M = _matrix(te_gpu, n, 3, 1, False)
    rng = np.random.default_rng(3)
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    v /= np.linalg.norm(v)
    ref = _run(te_gpu, M, v, 0, 1, 1.0)
    for fixed in (1, 0):
        ev = te_gpu.Evolver(M, v, 12.0, 3.0, [], tol=TOL, m=24)
        ev.set_option(te_gpu.OPT_FIXED_SPMV, fixed)
        ev.set_option(te_gpu.OPT_BARRIER_SPIN_LIMIT, 1 << 12)
        ev.set_option(te_gpu.OPT_BARRIER_EXTRA_ARRIVALS, 1)
        with pytest.raises(te_gpu.TeError) as e:
            ev.time_evolve()
        assert e.value.code == -10
        ev.set_option(te_gpu.OPT_BARRIER_EXTRA_ARRIVALS, 0)
        ev.reset(v)
        out = ev.time_evolve()
        assert out["n_steps"] == ref["n_steps"]
        assert np.linalg.norm(out["state"] - ref["state"]) < 2 * TOL
        ev.close()
