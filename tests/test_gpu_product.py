"""te_matrix_spmv on the caller's vectors against the product on sorted copies.

A product whose output overlaps its input, and one of a large real matrix,
reads a sorted copy of the input; any other reads and writes the caller's
vectors through the permutation, with the loads fetched ahead where the longest
row decides.  All sum each row in the same order, so the results are equal bit
for bit; against SciPy they agree to (row length + 2) roundings of the row's
sum of magnitudes.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, longest, giant, complex_values, seed):
    """Row lengths falling from `longest`, in random order; one row of `giant` entries."""
    rng = np.random.default_rng(seed)
    length = np.minimum(np.maximum(longest // np.arange(1, n + 1), rng.integers(0, 4, n)), n)
    length[0] = min(longest, n)
    if giant:
        length[-1] = giant
    length = rng.permutation(length)
    row = np.repeat(np.arange(n), length)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in length])
    val = rng.standard_normal(len(row)) + 1j * (rng.standard_normal(len(row)) if complex_values else 0.0)
    return row, col, val


@pytest.mark.parametrize("complex_values", [False, True])
@pytest.mark.parametrize("n,longest,giant,lanes", [
    (1, 1, 0, 0), (31, 7, 0, 0), (33, 8, 0, 0), (1000, 31, 0, 0),
    (1000, 32, 0, 0), (1001, 33, 0, 0), (2000, 47, 0, 0), (3000, 200, 0, 0),  # one more group, leftovers
    (70001, 33, 0, 0), (70001, 900, 0, 0),  # either side of the rule on the longest row
    (262144, 3, 0, 0), (262145, 3, 0, 0), (2097153, 3, 0, 0),  # real values: sorted input; all: sorted copies
    (5000, 40, 4500, 0), (20000, 40, 15000, 0),  # a long row by a warp; one in several segments
    (3000, 200, 0, 2), (3000, 33, 0, 4)])
def test_product_forms(te_gpu, n, longest, giant, lanes, complex_values):
    torch = pytest.importorskip("torch")
    from scipy import sparse
    row, col, val = _matrix(n, longest, giant, complex_values, n + longest)
    M = te_gpu.Matrix(n, row, col, val)
    if lanes:
        M.set_spmv_lanes(lanes)
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    alpha = 0.25 - 1.5j
    A = sparse.csr_matrix((val, (row, col)), shape=(n, n))
    exact = alpha * (A @ x)
    terms = np.maximum(np.bincount(row, minlength=n), 1) + 2
    bound = 4 * np.finfo(float).eps * terms * (abs(alpha) * (abs(A) @ abs(x))) + 1e-300

    for name in ("te_matrix_spmv", "te_matrix_spmv_noalloc")[:2 if n <= 1 << 18 else 1]:
        def product(src, dst):
            rc = getattr(te_gpu.lib(), name)(M.handle, alpha.real, alpha.imag, ctypes.c_void_p(src.data_ptr()),
                                             ctypes.c_void_p(dst.data_ptr()), None)
            assert rc == 0, te_gpu.lib().te_last_error()
            torch.cuda.synchronize()
            return dst.cpu().numpy().view(np.complex128).copy()

        def vector():
            return torch.from_numpy(x.view(np.float64).copy()).cuda()

        y = product(vector(), torch.full((2 * n,), float("nan"), dtype=torch.float64, device="cuda"))
        assert np.all(np.abs(y - exact) <= bound)
        same = vector()
        assert np.array_equal(product(same, same), y)
        shifted = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")  # the output one entry further
        shifted[:2 * n] = vector()
        assert np.array_equal(product(shifted[:2 * n], shifted[2:]), y)
        if name == "te_matrix_spmv":  # under capture: the pool's memory becomes the graph's
            graph, src, dst = torch.cuda.CUDAGraph(), vector(), torch.zeros(2 * n, dtype=torch.float64, device="cuda")
            with torch.cuda.graph(graph):
                rc = te_gpu.lib().te_matrix_spmv(M.handle, alpha.real, alpha.imag, ctypes.c_void_p(src.data_ptr()),
                                                 ctypes.c_void_p(dst.data_ptr()),
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == 0, te_gpu.lib().te_last_error()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(dst.cpu().numpy().view(np.complex128), y)


def test_product_scratch_is_given_back(te_gpu):
    """The pool's memory returns to the device with the buffer cache, and a
    cap of 0 keeps none."""
    torch = pytest.importorskip("torch")
    n = (1 << 18) + 1
    M = te_gpu.Matrix(n, np.arange(n), np.arange(n), np.ones(n, dtype=np.complex128))
    x, y = (torch.ones(2 * n, dtype=torch.float64, device="cuda") for _ in range(2))

    def product():
        rc = te_gpu.lib().te_matrix_spmv(M.handle, 1.0, 0.0, ctypes.c_void_p(x.data_ptr()),
                                         ctypes.c_void_p(y.data_ptr()), None)
        assert rc == 0, te_gpu.lib().te_last_error()
        torch.cuda.synchronize()

    product()
    te_gpu.release_buffers()
    free = torch.cuda.mem_get_info()[0]
    product()
    assert torch.cuda.mem_get_info()[0] <= free - 16 * n
    te_gpu.release_buffers()
    assert torch.cuda.mem_get_info()[0] == free
    try:
        te_gpu.set_buffer_cache_limit(0)
        product()
        assert torch.cuda.mem_get_info()[0] == free
    finally:
        te_gpu.set_buffer_cache_limit(8 << 30)
