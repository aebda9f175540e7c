"""Work that a user has this library do, as cases that can be timed and compared.

Every case is a dict of plain values.  ``prepare`` makes what a user's program
holds before the call (matrices, an evolver, a batch, start vectors), ``run``
makes one pass through the public entry points and returns its outputs whole,
``work`` counts what the pass cannot do without, ``exact`` computes the same
outputs in 64 bits with torch and numpy alone.

Kinds:
  chain     exp(-iHt)v on an open Bose-Hubbard chain, evolver kept, start vector
            on the GPU, occupations sampled on the way (the library's main use)
  call      one call with everything on the host (COO arrays, observables that
            are not diagonal, the overlap with the start vector)
  sparse    exp(-iHt)v under a complex Hermitian matrix with Zipf row lengths
            and random columns, handed over as a CSR that is already on the GPU
  batch     many chains of uneven length advanced together
  adjoint   loss and gradient of <n_0(T)> with respect to all couplings
  product   y = alpha H x on device buffers
"""
import ctypes
import math

import numpy as np
import torch

import timeevolver_gb300 as te
from timeevolver_gb300 import models

# sites, bosons, hopping, interaction, times and tolerances are those of the
# tests and of bench.py; the adjoint's couplings J_b ~ U(0.8, 1.2) are used for
# every chain that starts from a Fock state
DRAW_KINDS = ("chain", "call", "sparse", "batch", "adjoint", "product")


def listed():
    return [
        # the smallest evolutions: a parameter scan over short chains, where launches and waits count
        dict(name="chain_l6", kind="chain", L=6, N=6, U=2.0, t=10.0, dt=0.1, tol=1e-8, m=30, n_obs=6, start="fock",
             reorth=False),
        # the usual small run: every occupation sampled densely
        dict(name="chain_l8", kind="chain", L=8, N=8, U=3.0, t=10.0, dt=0.1, tol=1e-8, m=40, n_obs=8, start="fock",
             reorth=False),
        # a middle size at the tolerance of gradient work
        dict(name="chain_l10", kind="chain", L=10, N=10, U=2.0, t=5.0, dt=0.5, tol=1e-10, m=40, n_obs=10,
             start="fock", reorth=False),
        # the headline workload of bench.py
        dict(name="chain_l12", kind="chain", L=12, N=12, U=3.0, t=10.0, dt=0.5, tol=1e-8, m=40, n_obs=1,
             start="random", reorth=False),
        # the reorthogonalising mode, for results that must repeat across machines; an odd filling
        dict(name="chain_l9_reorth", kind="chain", L=9, N=8, U=2.0, t=2.0, dt=0.25, tol=1e-10, m=40, n_obs=9,
             start="random", reorth=True),
        # one call from host arrays: complex hopping, two bond currents, one bond energy, return amplitude
        dict(name="call_flux_l9", kind="call", L=9, N=9, U=1.0, phase=0.4, t=4.0, dt=0.1, tol=1e-10, m=40),
        # large irregular matrices; the second is the largest call (column blocks)
        dict(name="sparse_1e6", kind="sparse", n=1_000_003, exponent=1.5, max_len=256, t=100.0, dt=25.0, tol=1e-8,
             m=40),
        dict(name="sparse_8e6", kind="sparse", n=8_000_000, exponent=1.5, max_len=256, t=100.0, dt=100.0, tol=1e-8,
             m=40),
        # uneven chains together, as bench.py's batched workload
        dict(name="batch_48", kind="batch", count=48, l_min=6, l_max=10, t_max=10.0, tol=1e-10, m=32),
        # a gradient step of a control or fitting loop
        dict(name="adjoint_l10", kind="adjoint", L=10, N=10, U=2.0, t=5.0, tol=1e-10, m=40, interval=0.5, nodes=16),
        # single products, the building block of users' own solvers
        dict(name="product_l8", kind="product", L=8, N=8, U=3.0, matrix="chain"),
        dict(name="product_l12", kind="product", L=12, N=12, U=3.0, matrix="chain"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(DRAW_KINDS)
    u = round(rng.uniform(0.5, 4.0), 3)
    if kind == "chain":
        L = rng.randint(5, 12)
        N = max(3, L - rng.randint(0, 2))
        big = math.comb(N + L - 1, N) > 60_000
        reorth = (not big) and rng.random() < 0.3
        start = "random" if big or rng.random() < 0.5 else "fock"
        dt = rng.choice((0.05, 0.1, 0.25, 0.5))
        steps = rng.randint(2, 40)
        t = min(steps * dt, 2.0 if big or reorth else 10.0)
        t = dt * max(1, round(t / dt))
        return dict(kind=kind, L=L, N=N, U=u, t=t, dt=dt, tol=rng.choice((1e-8, 1e-10)), m=rng.randint(20, 48),
                    n_obs=rng.randint(0, min(L, 4 if big else L)), start=start, reorth=reorth)
    if kind == "call":
        L = rng.randint(5, 10)
        dt = rng.choice((0.05, 0.1, 0.2))
        return dict(kind=kind, L=L, N=max(3, L - rng.randint(0, 2)), U=u, phase=round(rng.uniform(0.0, 1.5), 3),
                    t=dt * rng.randint(4, 30), dt=dt, tol=1e-10, m=rng.randint(24, 44))
    if kind == "sparse":
        return dict(kind=kind, n=_log_int(rng, 70_000, 7_000_000), exponent=1.5, max_len=rng.choice((64, 200, 256)),
                    t=rng.choice((20.0, 100.0)), dt=rng.choice((5.0, 20.0)), tol=1e-8, m=rng.randint(24, 44))
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 4, 48), l_min=rng.randint(5, 7), l_max=rng.randint(8, 10),
                    t_max=round(rng.uniform(1.0, 8.0), 2), tol=1e-10, m=rng.randint(24, 40))
    if kind == "adjoint":
        L = rng.randint(6, 10)
        return dict(kind=kind, L=L, N=max(4, L - rng.randint(0, 1)), U=u, t=rng.choice((1.0, 2.5, 5.0)), tol=1e-10,
                    m=rng.randint(30, 44), interval=0.5, nodes=rng.choice((12, 16)))
    if rng.random() < 0.5:
        L = rng.randint(4, 12)
        return dict(kind="product", L=L, N=max(3, L - rng.randint(0, 3)), U=u, matrix="chain")
    return dict(kind="product", n=_log_int(rng, 1_000, 4_000_000), exponent=1.5, max_len=rng.choice((64, 200, 256)),
                matrix="sparse")


# ------------------------------------------------------------------ inputs

def _couplings(case, seed):
    """Bond hoppings: 1 for random start vectors (the headline), else U(0.8, 1.2)."""
    L = case["L"]
    if case.get("start") == "random" or case["kind"] == "product":
        return [1.0] * (L - 1)
    return list(np.random.default_rng(seed).uniform(0.8, 1.2, L - 1))


def _random_vector(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(n, 2, dtype=torch.float64, device="cuda", generator=g)
    return torch.view_as_complex(v / torch.linalg.vector_norm(v))


def _start_vector(case, n, seed):
    if case.get("start") == "fock":
        v = torch.zeros(n, dtype=torch.complex128, device="cuda")
        v[te.state_index_device(case["N"], [case["N"]] + [0] * (case["L"] - 1))] = 1.0
        return v
    return _random_vector(n, seed)


def _zipf_csr(case, seed):
    """H = (A + A^H) / 2 / (2 sqrt(max_len)): rows of A with Zipf lengths in
    [2, max_len], uniform columns, N(0, 1) real and imaginary parts.  A column
    drawn twice in a row stays two entries (they add)."""
    n, top = case["n"], case["max_len"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.arange(2, top + 1, dtype=torch.float64, device="cuda") ** -case["exponent"]
    cdf = torch.cumsum(p, 0) / p.sum()
    k = 2 + torch.searchsorted(cdf, torch.rand(n, dtype=torch.float64, device="cuda", generator=g)).clamp_(max=top - 2)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), k)
    col = torch.randint(0, n, (row.numel(),), device="cuda", generator=g)
    val = torch.view_as_complex(torch.randn(row.numel(), 2, dtype=torch.float64, device="cuda", generator=g))
    val *= 0.5 / (2.0 * math.sqrt(top))
    key = torch.cat([row * n + col, col * n + row])
    val = torch.cat([val, val.conj()])
    del row, col
    key, order = torch.sort(key, stable=True)
    val = val[order]
    del order
    row_ptr = torch.searchsorted(key, torch.arange(n + 1, device="cuda") * n).to(torch.int32)
    return row_ptr, (key % n).to(torch.int32), val.contiguous()


def _flux_terms(case, seed):
    """Chain with hopping -J_b e^{i phase}, and its observables' terms: the
    currents over the first and the middle bond, and the first bond's energy."""
    L, z = case["L"], complex(math.cos(case["phase"]), math.sin(case["phase"]))
    J = _couplings(case, seed)
    hop = [[models.lin_interaction(b, b + 1, 0, 0, False, -J[b] * z),
            models.lin_interaction(b, b + 1, 0, 0, True, -J[b] * z.conjugate())] for b in range(L - 1)]
    terms = [x for h in hop for x in h] + models.bose_hubbard_terms(L, [0.0] * (L - 1), case["U"])[2 * (L - 1):]

    def current(b):
        return [models.lin_interaction(b, b + 1, 0, 0, False, 1j * J[b] * z),
                models.lin_interaction(b, b + 1, 0, 0, True, -1j * J[b] * z.conjugate())]

    return terms, [current(0), current((L - 1) // 2), hop[0]]


def _batch_specs(case, seed):
    rng = np.random.default_rng(seed)
    span = case["l_max"] - case["l_min"] + 1  # every length alike: the batch's total size is the case's
    return [dict(L=case["l_min"] + i % span, J=float(rng.uniform(0.5, 1.5)),
                 U=float(rng.uniform(0.5, 4.0)), t=float(rng.uniform(0.25, 1.0) * case["t_max"]))
            for i in range(case["count"])]


def _chain_matrix(case, seed):
    return models.bose_hubbard_device(case["L"], case["N"], _couplings(case, seed), case["U"])


def _occupations_device(L, N, count):
    return [te.Matrix.from_terms_device(N, L, [models.number_operator(i, 1.0)])[0] for i in range(count)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        H, n = _chain_matrix(case, seed)
        v = _start_vector(case, n, seed)
        obs = _occupations_device(case["L"], case["N"], case["n_obs"])
        ev = te.Evolver(H, v.cpu().numpy(), case["t"], case["dt"], [("sparse", o) for o in obs], tol=case["tol"],
                        m=case["m"], reorth=case["reorth"])
        return dict(kind=kind, H=H, v=v, ev=ev)
    if kind == "call":
        B = models.Basis(case["N"], case["L"])
        terms, obs = _flux_terms(case, seed)
        v = np.zeros(len(B), dtype=np.complex128)
        v[B.index([case["N"]] + [0] * (case["L"] - 1))] = 1.0
        return dict(kind=kind, H=models.operator_matrix(terms, B), v=v, case=case,
                    obs=[("sparse", models.operator_matrix(o, B)) for o in obs] + [("vector", v)])
    if kind == "sparse":
        csr = _zipf_csr(case, seed)
        H = te.Matrix.from_device_csr(case["n"], *csr)
        del csr
        v = _random_vector(case["n"], seed + 1)
        torch.cuda.empty_cache()
        ev = te.Evolver(H, v.cpu().numpy(), case["t"], case["dt"], [], tol=case["tol"], m=case["m"])
        return dict(kind=kind, H=H, v=v, ev=ev)
    if kind == "batch":
        inst, number = [], {}
        for s in _batch_specs(case, seed):
            L = s["L"]
            H, n = models.bose_hubbard_device(L, L, s["J"], s["U"])
            if L not in number:
                number[L] = _occupations_device(L, L, 1)[0]
            v = np.zeros(n, dtype=np.complex128)
            v[te.state_index_device(L, [L] + [0] * (L - 1))] = 1.0
            inst.append(dict(H=H, v=v, t=s["t"], sampling_step=s["t"], tol=case["tol"], m=case["m"],
                             observables=[number[L]]))
        return dict(kind=kind, batch=te.Batch(inst))
    if kind == "adjoint":
        L, N = case["L"], case["N"]
        terms = []
        for b in range(L - 1):
            terms.append(te.Matrix.from_terms_device(N, L, [models.lin_interaction(b, b + 1, 0, 0, False, -1.0),
                                                            models.lin_interaction(b, b + 1, 0, 0, True, -1.0)])[0])
        inter = models.bose_hubbard_terms(L, [0.0] * (L - 1), 1.0)[2 * (L - 1):]
        H, n = te.Matrix.from_terms_device(N, L, inter)
        terms.append(H)
        v = np.zeros(n, dtype=np.complex128)
        v[te.state_index_device(N, [N] + [0] * (L - 1))] = 1.0
        adj = te.Adjoint(terms, _occupations_device(L, N, 1)[0], v, T=case["t"], tol=case["tol"], m=case["m"],
                         checkpoint_interval=case["interval"], nodes_per_interval=case["nodes"])
        return dict(kind=kind, adj=adj, theta=np.array(_couplings(case, seed) + [case["U"]]))
    if case["matrix"] == "chain":
        H, n = _chain_matrix(case, seed)
    else:
        n = case["n"]
        H = te.Matrix.from_device_csr(n, *_zipf_csr(case, seed))
    x = _random_vector(n, seed + 1)
    return dict(kind="product", H=H, x=x, y=torch.empty_like(x))


def run(state):
    kind = state["kind"]
    if kind in ("chain", "sparse"):
        ev = state["ev"]
        ev.reset(None, device_ptr=state["v"].data_ptr())
        r = ev.time_evolve()
        return dict(samples=r["samples"], state=r["state"], num_samples=r["num_samples"])
    if kind == "call":
        c = state["case"]
        r = te.evolve(state["H"], state["v"], c["t"], c["dt"], state["obs"], tol=c["tol"], m=c["m"])
        return dict(samples=r["samples"], state=r["state"], num_samples=r["num_samples"])
    if kind == "batch":
        b = state["batch"]
        res = b.run()
        return dict(samples=np.concatenate([b.samples(i) for i in range(b.B)]),
                    state=np.concatenate([b.state(i) for i in range(b.B)]),
                    num_samples=np.array([r["num_samples"] for r in res]))
    if kind == "adjoint":
        loss, grad = state["adj"].run(state["theta"])
        return dict(loss=loss, grad=grad)
    y = state["y"]
    rc = te.lib().te_matrix_spmv(state["H"].handle, 0.0, -1.0, ctypes.c_void_p(state["x"].data_ptr()),
                                 ctypes.c_void_p(y.data_ptr()), None)
    if rc != te.TE_OK:
        raise te.TeError(rc, "te_matrix_spmv")
    return y


# ------------------------------------------------------------ work and values

def _chain_size(L, N):
    """(dimension, stored entries) of an open chain: every bond moves a boson
    either way where its source site is not empty."""
    return math.comb(N + L - 1, N), math.comb(N + L - 1, N) + 2 * (L - 1) * math.comb(N + L - 2, L - 1)


def _sparse_entries(case):
    k = np.arange(2, case["max_len"] + 1)
    p = k ** -case["exponent"]
    return 2.0 * case["n"] * float(np.sum(k * p) / np.sum(p))


def _evolution(n, nnz, value_bytes, degree, samples, n_obs):
    """A polynomial of H of the degree that t and the spectrum ask for: per
    degree the matrix once and the vector read and written; per sample the
    state and its observables."""
    spmv = nnz * (value_bytes + 4) + 32 * n
    flops = nnz * value_bytes / 2
    return {"bytes": degree * spmv + samples * (16 + 8 * n_obs) * n,
            "flops": degree * flops + samples * n * (4 + 2 * n_obs)}


def _chain_degree(L, N, U, t):
    """t times half the spectral width (interaction energies 0 .. U N (N - 1) / 2
    and at most 2 per boson from hopping), plus the tail of the expansion."""
    return math.ceil(t * (U * N * (N - 1) / 4.0 + 2.0 * N)) + 10


def work(case):
    kind = case["kind"]
    if kind == "chain" or kind == "call":
        n, nnz = _chain_size(case["L"], case["N"])
        complex_h = kind == "call"
        return _evolution(n, nnz, 16 if complex_h else 8, _chain_degree(case["L"], case["N"], case["U"], case["t"]),
                          int(case["t"] / case["dt"] + 1e-9) + 1, 4 if complex_h else case["n_obs"])
    if kind == "sparse":
        return _evolution(case["n"], _sparse_entries(case), 16, math.ceil(case["t"]) + 10,
                          int(case["t"] / case["dt"] + 1e-9) + 1, 0)
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["count"]):
            L = case["l_min"] + i % (case["l_max"] - case["l_min"] + 1)
            n, nnz = _chain_size(L, L)
            w = _evolution(n, nnz, 8, _chain_degree(L, L, 2.25, 0.625 * case["t_max"]), 2, 1)
            for k in total:
                total[k] += w[k]
        return total
    if kind == "adjoint":
        n, nnz = _chain_size(case["L"], case["N"])
        nodes = math.ceil(case["t"] / case["interval"]) * case["nodes"]
        w = _evolution(n, nnz, 8, _chain_degree(case["L"], case["N"], case["U"], case["t"]), nodes, 0)
        # forward and costate, then one bilinear pass over both states of every node
        return {"bytes": 2 * w["bytes"] + 32 * n * nodes + 12 * nnz, "flops": 2 * w["flops"] + 8 * nnz * nodes}
    if case["matrix"] == "chain":
        n, nnz = _chain_size(case["L"], case["N"])
        return {"bytes": 12 * nnz + 32 * n, "flops": 4 * nnz}
    nnz = _sparse_entries(case)
    return {"bytes": 20 * nnz + 32 * case["n"], "flops": 8 * nnz}


def _occupations(L, N):
    """Occupation vectors of the chain in the library's basis order: mode by
    mode from the last to the second, every non-empty filling of that mode is
    appended to the states found so far; the first mode takes the rest."""
    s = np.zeros((1, L), dtype=np.int64)
    for k in range(L - 1, 0, -1):
        room = N - s.sum(axis=1)
        parent = np.repeat(np.arange(len(s)), room)
        new = s[parent].copy()
        new[:, k] = 1 + np.arange(len(parent)) - np.repeat(np.cumsum(room) - room, room)
        s = np.concatenate([s, new])
    s[:, 0] = N - s.sum(axis=1)
    return torch.from_numpy(s).cuda()


def _hops(s, b):
    """(row, col, amplitude) of a_{b+1}^dag a_b on every state."""
    base = (int(s.max()) + 1) ** torch.arange(s.shape[1], device="cuda")
    keys, order = torch.sort((s * base).sum(1))
    src = torch.nonzero(s[:, b] > 0)[:, 0]
    moved = s[src].clone()
    moved[:, b] -= 1
    moved[:, b + 1] += 1
    dst = order[torch.searchsorted(keys, (moved * base).sum(1))]
    return dst, src, torch.sqrt((s[src, b] * (s[src, b + 1] + 1)).double())


def _csr(n, row, col, val):
    key, order = torch.sort(row * n + col)
    ptr = torch.searchsorted(key, torch.arange(n + 1, device="cuda") * n)
    return torch.sparse_csr_tensor(ptr, key % n, val[order], size=(n, n))


def _chain_operator(s, amps, diag):
    """sum_b amps[b] a_{b+1}^dag a_b + h.c. + diag (a_b^dag a_{b+1} has the conjugate amplitude).
    The library's matrices hold an operator's amplitude from state i to state j at (i, j)."""
    n = len(s)
    row, col, val = [torch.arange(n, device="cuda")], [torch.arange(n, device="cuda")], [diag.to(torch.complex128)]
    for b, a in enumerate(amps):
        if a == 0:
            continue
        r, c, w = _hops(s, b)
        row += [c, r]
        col += [r, c]
        val += [w * complex(a), w * complex(a).conjugate()]
    return _csr(n, torch.cat(row), torch.cat(col), torch.cat(val))


def _interval(H):
    """Gershgorin bounds of the spectrum."""
    ptr, col, val = H.crow_indices(), H.col_indices(), 1.0 * H.values()
    n = H.shape[0]
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), ptr[1:] - ptr[:-1])
    d = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, torch.where(row == col, val.real, 0.0))
    r = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, row, torch.where(row == col, 0.0, val.abs()))
    return float((d - r).min()), float((d + r).max())


class _Propagator:
    """exp(-i H t) v by the Chebyshev expansion, coefficients by an FFT of the
    generating function; the spectrum from Gershgorin (or the given bound)."""

    def __init__(self, H, bounds=None):
        lo, hi = bounds or _interval(H)
        self.H, self.c, self.r, self.known = H, 0.5 * (lo + hi), 0.5 * (hi - lo) * 1.0001 + 1e-12, {}

    def _coefficients(self, t):
        if t not in self.known:
            z = t * self.r
            m = 1 << int(math.ceil(math.log2(2 * abs(z) + 200)))
            f = np.fft.fft(np.exp(-1j * z * np.cos(2 * np.pi * np.arange(m) / m))) / m
            k = int(np.max(np.nonzero(np.abs(f[:m // 2]) > 2e-16)[0])) + 1
            f = 2 * f[:k]
            f[0] *= 0.5
            self.known[t] = f * np.exp(-1j * t * self.c)
        return self.known[t]

    def __call__(self, v, t):
        f = self._coefficients(t)
        a, out = v, v * complex(f[0])
        if len(f) > 1:
            b = (self.H @ v - self.c * v) / self.r
            out += b * complex(f[1])
            for x in f[2:]:
                a, b = b, (self.H @ b - self.c * b) * (2.0 / self.r) - a
                out += b * complex(x)
        return out


def _trajectory(U, v, t, dt, observe):
    """Observables at 0, dt, ... <= t and the last state."""
    count = int(math.floor(t / dt)) + 1
    rows = [observe(v)]
    for _ in range(count - 1):
        v = U(v, dt)
        rows.append(observe(v))
    return torch.tensor(rows, dtype=torch.float64).reshape(count, len(rows[0])).T.contiguous(), v


def _expect(O, v):
    return float(torch.vdot(v, O @ v).real)


def _interaction(s, U):
    return 0.5 * U * (s * (s - 1)).sum(1).double()


def _fock_index(s, N):
    return int(torch.nonzero(s[:, 0] == N)[0])


def _exact_adjoint(case, s, theta):
    L, N = case["L"], case["N"]
    n = len(s)
    H = _chain_operator(s, [-x for x in theta[:L - 1]], _interaction(s, theta[L - 1]))
    parts = [_chain_operator(s, [-1.0 if k == b else 0.0 for k in range(L - 1)],
                             torch.zeros(n, dtype=torch.float64, device="cuda")) for b in range(L - 1)]
    w_int = _interaction(s, 1.0)
    U = _Propagator(H)
    v = torch.zeros(n, dtype=torch.complex128, device="cuda")
    v[_fock_index(s, N)] = 1.0
    pieces = int(math.ceil(case["t"] / case["interval"]))
    x, w = np.polynomial.legendre.leggauss(case["nodes"])
    h = case["t"] / pieces
    times = np.concatenate([h * (k + 0.5 + 0.5 * x) for k in range(pieces)])
    weights = np.concatenate([0.5 * h * w] * pieces)
    psi, now, states = v, 0.0, []
    for t in times:
        psi, now = U(psi, float(t - now)), t
        states.append(psi)
    psi = U(psi, float(case["t"] - now))
    n0 = s[:, 0].double()
    loss = float((n0 * psi.abs().square()).sum())
    lam, now, grad = n0 * psi, case["t"], np.zeros(L)
    for t, wt, ps in zip(times[::-1], weights[::-1], states[::-1]):
        lam, now = U(lam, float(t - now)), t
        for k, P in enumerate(parts):
            grad[k] += 2.0 * wt * float(torch.vdot(lam, P @ ps).imag)
        grad[L - 1] += 2.0 * wt * float(torch.vdot(lam, w_int * ps).imag)
    return dict(loss=loss, grad=grad)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sparse" or case.get("matrix") == "sparse":
        ptr, col, val = _zipf_csr(case, seed)
        H = torch.sparse_csr_tensor(ptr, col, val, size=(case["n"], case["n"]))
        v = _random_vector(case["n"], seed + 1)
        if kind == "product":
            return -1j * (H @ v)
        samples, v = _trajectory(_Propagator(H), v, case["t"], case["dt"], lambda x: [])
        return dict(samples=samples, state=v.cpu().numpy(), num_samples=None)
    if kind == "batch":
        samples, states = [], []
        for sp in _batch_specs(case, seed):
            s = _occupations(sp["L"], sp["L"])
            H = _chain_operator(s, [-sp["J"]] * (sp["L"] - 1), _interaction(s, sp["U"]))
            v = torch.zeros(len(s), dtype=torch.complex128, device="cuda")
            v[_fock_index(s, sp["L"])] = 1.0
            n0 = s[:, 0].double()
            o, v = _trajectory(_Propagator(H), v, sp["t"], sp["t"], lambda x: [float((n0 * x.abs().square()).sum())])
            samples.append(o)
            states.append(v)
        return dict(samples=torch.cat(samples), state=torch.cat(states).cpu().numpy(), num_samples=None)
    L, N = case["L"], case["N"]
    s = _occupations(L, N)
    n = len(s)
    J = _couplings(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, s, np.array(J + [case["U"]]))
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    if kind == "call":
        z = complex(math.cos(case["phase"]), math.sin(case["phase"]))
        # the term -J_b z a_b^dag a_{b+1} is the conjugate partner of _hops' direction
        H = _chain_operator(s, [-x * z.conjugate() for x in J], _interaction(s, case["U"]))

        def one(b, a):
            return _chain_operator(s, [a if k == b else 0.0 for k in range(L - 1)], zero)

        mid = (L - 1) // 2
        obs = [one(0, -1j * J[0] * z.conjugate()), one(mid, -1j * J[mid] * z.conjugate()),
               one(0, -J[0] * z.conjugate())]
        v0 = torch.zeros(n, dtype=torch.complex128, device="cuda")
        v0[_fock_index(s, N)] = 1.0
        samples, v = _trajectory(_Propagator(H), v0, case["t"], case["dt"],
                                 lambda x: [_expect(O, x) for O in obs] + [float(torch.vdot(x, v0).abs() ** 2)])
        return dict(samples=samples, state=v.cpu().numpy(), num_samples=None)
    H = _chain_operator(s, [-x for x in J], _interaction(s, case["U"]))
    if kind == "product":
        return -1j * (H @ _random_vector(n, seed + 1))
    if case.get("start") == "fock":
        v = torch.zeros(n, dtype=torch.complex128, device="cuda")
        v[_fock_index(s, N)] = 1.0
    else:
        v = _random_vector(n, seed)
    occ = s[:, :case["n_obs"]].double()
    samples, v = _trajectory(_Propagator(H), v, case["t"], case["dt"],
                             lambda x: [] if not case["n_obs"] else (x.abs().square() @ occ).tolist())
    return dict(samples=samples, state=v.cpu().numpy(), num_samples=None)
