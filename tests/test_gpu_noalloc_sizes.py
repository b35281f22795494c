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
