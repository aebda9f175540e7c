"""The one-launch Lanczos kernels of te_resident.cu (70 001 rows: in registers;
400 001: streamed) where their scales, their exits and their range end; needs a
GB300.

The matrices are open chains, whose exact evolutions SciPy gives in 64 bits.
"""
import threading

import numpy as np
import pytest
import scipy.linalg
import scipy.sparse
import scipy.sparse.linalg

pytestmark = pytest.mark.gpu

TOL = 1e-9
RESIDENT, STREAMED = 70_001, 400_001
FORMS = [(RESIDENT, 1), (RESIDENT, 0), (STREAMED, 1)]  # rows, TE_OPT_FIXED_SPMV


def _tridiagonal(n, seed):
    """Real diagonal in [-1, 1], hopping in [0.5, 1]."""
    rng = np.random.default_rng(seed)
    return rng.uniform(-1.0, 1.0, n), rng.uniform(0.5, 1.0, n - 1)


def _scipy(diag, hop):
    return scipy.sparse.diags_array([diag, hop, hop], offsets=[0, 1, -1], format="csr")


def _matrix(te, diag, hop):
    A = _scipy(diag, hop).tocsr()
    A.eliminate_zeros()
    return te.Matrix.from_csr(len(diag), A.indptr, A.indices, A.data.astype(np.complex128))


def _evolver(te, M, v, t, fused, fixed, exp_factor=1.0, tol=TOL, m=24):
    ev = te.Evolver(M, v, t, t, [], exp_factor=exp_factor, tol=tol, m=m)
    ev.set_option(te.OPT_FUSED_LANCZOS, fused)
    ev.set_option(te.OPT_FIXED_SPMV, fixed)
    return ev


def _run(*args, **kw):
    ev = _evolver(*args, **kw)
    out = ev.time_evolve(trace=True)
    ev.close()
    return out


def _random(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return v / np.linalg.norm(v)


@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("energy", [1e1, 1e4, 1e6, 1e9])
@pytest.mark.parametrize("n,fixed", FORMS)
def test_large_energy_out_of_reach(te_gpu, n, fixed, energy, local):
    """||H|| far above what the state reaches (the last row couples to no other
    and holds no weight): both ways carry the vectors with the same number of
    bits, so the same roundings in another order; their errors are random sums
    of as many terms of the same size."""
    diag, hop = _tridiagonal(n, n)
    diag[-1], hop[-1] = energy, 0.0
    v = _random(n, 5)
    if local:
        v *= 1e-3
        v[n // 3] += 1.0
    v[-1] = 0.0
    v /= np.linalg.norm(v)
    M = _matrix(te_gpu, diag, hop)
    t = 1.5
    exact = np.append(scipy.sparse.linalg.expm_multiply(-1j * t * _scipy(diag[:-1], hop[:-1]), v[:-1]), 0.0)
    one, passes = (_run(te_gpu, M, v, t, fused, fixed, m=30) for fused in (1, 0))
    assert one["n_steps"] == passes["n_steps"] and passes["launches"] > one["launches"]
    assert [s["m_eff"] for s in one["trace"]] == [s["m_eff"] for s in passes["trace"]]
    error, other = (np.linalg.norm(out["state"] - exact) for out in (one, passes))
    assert error <= 2 * other + 1e-14


@pytest.mark.parametrize("exp_factor", [1.0, -0.7])
@pytest.mark.parametrize("length", [5, 24])
@pytest.mark.parametrize("n,fixed", FORMS)
def test_lucky_breakdown(te_gpu, n, fixed, length, exp_factor):
    """A start vector in an invariant subspace of `length` dimensions, fewer
    than the Krylov dimension or as many (the last iteration's breakdown)."""
    diag, hop = _tridiagonal(n, n)
    hop[length - 1] = 0.0
    v = np.zeros(n, dtype=np.complex128)
    v[0] = 1.0
    M = _matrix(te_gpu, diag, hop)
    t = 12.0
    block = np.diag(diag[:length]) + np.diag(hop[:length - 1], 1) + np.diag(hop[:length - 1], -1)
    exact = scipy.linalg.expm(-1j * exp_factor * t * block)[:, 0]
    one, passes = (_run(te_gpu, M, v, t, fused, fixed, exp_factor) for fused in (1, 0))
    assert passes["launches"] > one["launches"]
    assert one["n_steps"] == passes["n_steps"] and one["status"] == passes["status"]
    for a, b in zip(one["trace"], passes["trace"]):
        assert a["breakdown"] == b["breakdown"] and a["m_eff"] == b["m_eff"]
    assert one["trace"][0]["breakdown"] == 1 and one["trace"][0]["m_eff"] == length
    for out in (one, passes):
        assert np.linalg.norm(out["state"][:length] - exact) < TOL and not np.any(out["state"][length:])


@pytest.mark.parametrize("exp_factor", [0.6, -0.7])
@pytest.mark.parametrize("n,fixed", FORMS)
def test_sign_of_the_exponent(te_gpu, n, fixed, exp_factor):
    """Several steps of either sign against the exact state."""
    diag, hop = _tridiagonal(n, n)
    v = _random(n, 7)
    t = 12.0
    exact = scipy.sparse.linalg.expm_multiply(-1j * exp_factor * t * _scipy(diag, hop), v)
    out = _run(te_gpu, _matrix(te_gpu, diag, hop), v, t, 1, fixed, exp_factor)
    assert out["n_steps"] > 1
    assert np.linalg.norm(out["state"] - exact) < TOL


@pytest.mark.parametrize("start", ["row", "bound"])
@pytest.mark.parametrize("m", [30, 40, 41, 64])
@pytest.mark.parametrize("n,fixed", FORMS)
def test_krylov_dimensions(te_gpu, n, fixed, m, start):
    """One row as the start, and a chain with a bound state outside its band
    (its Ritz value converges within a step) on a random start, either side of
    the last Krylov dimension of the one-launch kernels."""
    diag, hop = _tridiagonal(n, n)
    v = _random(n, 9)
    if start == "row":
        v = np.zeros(n, dtype=np.complex128)
        v[n // 2] = 1.0
    else:
        diag[n // 3] = 20.0
        v[n // 3] += 0.5
        v /= np.linalg.norm(v)
    M = _matrix(te_gpu, diag, hop)
    t = 10.0
    exact = scipy.sparse.linalg.expm_multiply(-1j * t * _scipy(diag, hop), v)
    one, passes = (_run(te_gpu, M, v, t, fused, fixed, m=m) for fused in (1, 0))
    assert (passes["launches"] > one["launches"]) == (m <= 40)
    for out in (one, passes):
        assert np.linalg.norm(out["state"] - exact) < TOL


def test_two_threads(te_gpu):
    """Evolvers on two host threads, each launch as large as the GPU: the same
    states as one after the other, bit for bit."""
    jobs = []
    for n, fixed in ((RESIDENT, 1), (STREAMED, 1)):
        diag, hop = _tridiagonal(n, n)
        M, v = _matrix(te_gpu, diag, hop), _random(n, 3)
        jobs.append((M, _evolver(te_gpu, M, v, 12.0, 1, fixed), v, _run(te_gpu, M, v, 12.0, 1, fixed)["state"]))
    states = [[], []]

    def work(k):
        _, ev, v, _ = jobs[k]
        te_gpu.lib().te_set_device(0)
        for _ in range(5):
            ev.reset(v)
            states[k].append(ev.time_evolve()["state"])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for k, (_, ev, _, alone) in enumerate(jobs):
        assert len(states[k]) == 5 and all(np.array_equal(s, alone) for s in states[k])
        ev.close()


def test_streamed_exchange_timeout(te_gpu):
    """A wait of the streaming kernel that runs out: the error, and the same
    evolver then runs to the exact state."""
    diag, hop = _tridiagonal(STREAMED, STREAMED)
    M, v = _matrix(te_gpu, diag, hop), _random(STREAMED, 3)
    ev = _evolver(te_gpu, M, v, 3.0, 1, 1)
    ev.set_option(te_gpu.OPT_BARRIER_SPIN_LIMIT, 1 << 12)
    ev.set_option(te_gpu.OPT_BARRIER_EXTRA_ARRIVALS, 1)
    with pytest.raises(te_gpu.TeError) as e:
        ev.time_evolve()
    assert e.value.code == -10
    ev.set_option(te_gpu.OPT_BARRIER_EXTRA_ARRIVALS, 0)
    ev.reset(v)
    exact = scipy.sparse.linalg.expm_multiply(-3j * _scipy(diag, hop), v)
    assert np.linalg.norm(ev.time_evolve()["state"] - exact) < TOL
    ev.close()


@pytest.mark.parametrize("scale", [1e20, 1e100, 1e154, 1e200, 1e299])
@pytest.mark.parametrize("n,fixed", FORMS)
def test_overflow_is_an_error(te_gpu, n, fixed, scale):
    """The norms of the unnormalised basis grow with ||H||^m: beyond the range of
    a double the evolution ends with an error (no step size or no eigenvalues),
    not with a state."""
    diag, hop = _tridiagonal(n, n)
    M, v = _matrix(te_gpu, scale * diag, scale * hop), _random(n, 3)
    for fused in (1, 0):
        ev = _evolver(te_gpu, M, v, 1.0, fused, fixed)
        with pytest.raises(te_gpu.TeError) as e:
            ev.time_evolve()
        assert e.value.code in (-5, -6)
        ev.close()


@pytest.mark.parametrize("scale", [1e-6, 1e-5, 1e5])
@pytest.mark.parametrize("n", [RESIDENT, STREAMED])
def test_units_of_energy(te_gpu, n, scale):
    """The same evolution in other units; at 1e-6 the basis's squared norms leave
    the range of a double after 26 iterations, which ends the step as a lucky
    breakdown would."""
    diag, hop = _tridiagonal(n, n)
    M, v = _matrix(te_gpu, scale * diag, scale * hop), _random(n, 3)
    exact = scipy.sparse.linalg.expm_multiply(-3j * _scipy(diag, hop), v)
    for fused in (1, 0):
        out = _run(te_gpu, M, v, 3.0 / scale, fused, 1, m=40 if scale < 1e-5 else 28)
        assert np.linalg.norm(out["state"] - exact) < TOL


def test_same_route_in_every_run(te_gpu):
    """What a run finds on the matrix from earlier ones (timed lanes per row, a
    column-blocked fixed-point form) does not change its route: the same launches
    and the same state, bit for bit."""
    n, band = RESIDENT, 64  # rows long enough for several lanes each
    rng = np.random.default_rng(1)
    sides = [rng.standard_normal(n - k) / band for k in range(1, band)]
    A = scipy.sparse.diags_array(sides + sides, offsets=[*range(1, band), *range(-1, -band, -1)], format="csr")
    v = _random(n, 3)

    def matrix():
        return te_gpu.Matrix.from_csr(n, A.indptr, A.indices, A.data.astype(np.complex128))

    def run(M, fixed):
        out = _run(te_gpu, M, v, 3.0, 1, fixed)
        return out["launches"], out["state"]

    timed = matrix()
    timed.set_spmv_lanes(-1)
    runs = [run(timed, fixed) for fixed in (1, 0, 0, 1)]
    assert timed.spmv_lanes(tune=False) > 1
    for a, b in ((0, 3), (1, 2)):
        assert runs[a][0] == runs[b][0] and np.array_equal(runs[a][1], runs[b][1])
    blocked = matrix()
    before = run(blocked, 0)
    blocked.set_fixed_blocks(2)
    run(blocked, 1)
    after = run(blocked, 0)
    assert before[0] == after[0] and np.array_equal(before[1], after[1])
