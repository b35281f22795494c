"""One context per host thread: solvers whose launches differ in shared memory run side by side."""
import threading

import numpy as np
import pytest

import drops_gb300 as tf

pytestmark = pytest.mark.gpu


def band(m, half):
    """Symmetric, diagonally dominant, 2 half + 1 entries in a row."""
    i = np.arange(m)[:, None]
    cols = i + np.arange(-half, half + 1)[None, :]
    vals = np.where(cols == i, 2.0 * half + 0.5, -1.0)
    keep = (cols >= 0) & (cols < m)
    rp = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int64)
    return rp, cols[keep].astype(np.int64), vals[keep]


@pytest.mark.parametrize("solver", ["pcg", "gmres", "gmres mixed"])
def test_two_threads_two_sizes(solver):
    """Solves of two iterations, so that the host's part of a call is most of it: every call returns the status, the
    residual and the iterate of the first.  The blocks of both contexts (16 and 47) fit the device together; their
    shared memory differs by the 3 and 101 entries of a row."""
    rounds, errors, ready = 2000, [], threading.Barrier(2)

    def work(m, half):
        k = -1
        try:
            with tf.TraceFEM(0) as ctx:
                ctx.matrix_upload(*band(m, half))
                ctx.vec_upload(tf.VEC_B, np.random.default_rng(m).standard_normal(m))
                first = None
                for k in range(rounds):
                    ctx.vec_fill(tf.VEC_X, m, 0.0)
                    if k == 2:  # layouts built, later launches alike
                        ready.wait(60)
                    if solver == "pcg":
                        got = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=0.0, max_iter=2)
                    else:
                        prec = tf.PREC_MIXED if "mixed" in solver else tf.PREC_FP64
                        got = ctx.gmres_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, restart=10, tol=0.0, max_iter=2, precision=prec)
                    if k >= 1:  # the first PCG of a small pattern takes a cluster
                        now = (*got, ctx.vec_download(tf.VEC_X).tobytes())
                        assert first is None or now == first
                        first = now
        except Exception as e:
            errors.append((m, k, e))
            ready.abort()

    threads = [threading.Thread(target=work, args=a) for a in ((1024, 1), (3000, 50))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
