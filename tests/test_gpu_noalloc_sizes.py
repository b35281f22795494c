"""tf_pcg_jacobi_noalloc over sizes (one row to several per lane) and row lengths (1, 8 and 32 lanes per row)."""

import ctypes as C

import numpy as np
import pytest

import drops_gb300 as tf
from tests.test_gpu_pcg_cluster import cg, mul, spd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,links", [(1, lambda i: 0), (31, lambda i: 2), (33, lambda i: 2), (129, lambda i: 3),
                                     (20000, lambda i: i % 5), (600, lambda i: 24), (400, lambda i: 80),
                                     (700, lambda i: 300 if i in (5, 650) else 1)])
def test_sizes_and_row_lengths(m, links):
    tf.load_library()
    A = spd(m, links, seed=3)
    rp, ci, v, b = A
    its = cg(A, 1e-10)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rp.astype(np.int32), ci.astype(np.int32), v, b, np.zeros(m))]
    torch.cuda.synchronize()
    it, tol = C.c_int(10000), C.c_double(1e-10)
    st = tf.load_library().tf_pcg_jacobi_noalloc(C.c_int64(m), *[C.c_void_p(t.data_ptr()) for t in d], C.byref(it),
                                                 C.byref(tol), C.c_int(1), None)
    assert st == tf.OK and tol.value <= 1e-10 and abs(it.value - its) <= 1
    # well conditioned: the recursive residual follows the true one to a few ulps of |b|
    assert np.linalg.norm(b - mul(A, d[4].cpu().numpy())) <= 1.01e-10 * np.linalg.norm(b)


def bordered(m, half, border):
    """Band of 2 half + 1 entries with `border` dense rows and columns, symmetric and diagonally dominant."""
    import scipy.sparse as sp

    off = [k for k in range(-half, half + 1) if k]
    B = sp.diags([np.full(m - abs(k), -1.0) for k in off], off, shape=(m, m)).tolil()
    for k in range(border):
        r = m // 2 + 40 * k
        B[r, :] = -0.4 / m
        B[:, r] = -0.4 / m
    B.setdiag(0.0)
    B = B.tocsr()
    A = (B + sp.diags(0.5 - np.asarray(B.sum(axis=1)).ravel())).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data, np.random.default_rng(m).standard_normal(m)


@pytest.mark.parametrize("m,half,border", [(3000, 1, 1), (3000, 1, 2), (3000, 20, 1), (129, 1, 1), (130, 1, 1)])
def test_dense_rows(m, half, border):
    """Rows far above the mean (more than 128 entries on one lane, 1024 on eight) are summed by their warp."""
    A = bordered(m, half, border)
    its = cg(A, 1e-10)
    st, it, res, x, _ = solve(A)
    assert st == tf.OK and res <= 1e-10 and abs(it - its) <= 1
    # smallest eigenvalue 0.5: the recursive residual follows the true one
    assert np.linalg.norm(A[3] - mul(A, x)) <= 1.01e-10 * np.linalg.norm(A[3])


def test_dense_row_does_not_hold_up_the_grid():
    """65,536 rows of 3 entries with one dense row: its entries in 256 trips of a warp, each two dependent reads of L2 at
    about 0.5 us, make 0.3 ms per iteration; three times that is allowed.  (8,192 trips of one lane take 8 ms.)"""
    A = bordered(65536, 1, 1)
    best = min(solve(A, max_iter=20, tol=0.0)[4] for _ in range(3))
    assert best <= 20 * 0.9e-3


def solve(A, max_iter=10000, tol=1e-10):
    import time

    rp, ci, v, b = A
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rp.astype(np.int32), ci.astype(np.int32), v, b, np.zeros(len(b)))]
    torch.cuda.synchronize()
    it, t = C.c_int(max_iter), C.c_double(tol)
    t0 = time.perf_counter()
    st = tf.load_library().tf_pcg_jacobi_noalloc(C.c_int64(len(b)), *[C.c_void_p(a.data_ptr()) for a in d], C.byref(it),
                                                 C.byref(t), C.c_int(1), None)
    seconds = time.perf_counter() - t0
    return st, it.value, t.value, d[4].cpu().numpy(), seconds
