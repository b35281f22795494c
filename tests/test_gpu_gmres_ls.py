"""Two-grid-step MGS GMRES on general matrices: sizes around the slices and runs of its blocks, every side and restart."""
import numpy as np
import pytest

import drops_gb300 as tf
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-11


@pytest.fixture(scope="module")
def ctx():
    from drops_gb300 import build

    build.build()
    c = tf.TraceFEM()
    yield c
    c.close()


def banded(m, seed):
    """Nonsymmetric CSR matrix with diagonal 2 and off-diagonal row sums of absolute values at most 1, so
    |A^-1|_inf <= 1: entries at distance 1, 7 and m // 3."""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(m)], [np.arange(m)], [np.full(m, 2.0)]
    for d in {1, 7, max(m // 3, 1)}:
        for s in (d, -d):
            i = np.arange(max(0, -s), m - max(0, s))
            if i.size:
                rows.append(i)
                cols.append(i + s)
                vals.append(rng.uniform(-1.0, 1.0, i.size) / 6.0)
    rows, cols, vals = (np.concatenate(x) for x in (rows, cols, vals))
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int64)
    return rp, cols[o].astype(np.int64), vals[o], rng.standard_normal(m)


def solve(ctx, A, b, restart, method, prec):
    ctx.matrix_upload(*A)
    ctx.vec_upload(tf.VEC_B, b)
    ctx.vec_upload(tf.VEC_X, np.zeros(b.size))
    st, it, res = ctx.gmres_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, restart=restart, tol=TOL, method=method, precision=prec)
    assert st == tf.OK and res <= TOL
    return it, ctx.vec_download(tf.VEC_X)


@pytest.mark.parametrize("m", [1, 31, 33, 512, 513, 20011])
@pytest.mark.parametrize("restart,method,prec", [(2, 0, 0), (3, 1, 0), (50, 0, 0), (64, 1, 0), (64, 0, 0), (2, 0, 1),
                                                 (64, 0, 1)])
def test_gmres_sizes(ctx, m, restart, method, prec):
    """Both solvers stop at |r| <= TOL |b| (left: |D^-1 r| <= TOL |D^-1 b|, D = 2), and |A^-1|_inf <= 1, so the
    solutions differ by at most 2 TOL |b| in the maximum norm (10% more for the rounding of the residuals)."""
    rp, ci, v, b = banded(m, m + restart)
    it, x = solve(ctx, (rp, ci, v), b, restart, method, prec)
    _, ox, oit, _ = O.gmres_jacobi(rp, ci, v, b, restart=restart, tol=TOL, method=method)
    assert np.abs(x - ox).max() <= 2.2 * TOL * np.linalg.norm(b)
    if prec == tf.PREC_FP64:
        assert abs(it - oit) <= 2, (it, oit)


def test_gmres_run_beyond_shared_memory(ctx):
    """More rows per block than its shared memory holds (FP64, 1.7 million rows): w and v_i from global memory."""
    rp, ci, v, b = banded(1700000, 3)
    _, x = solve(ctx, (rp, ci, v), b, 10, 0, tf.PREC_FP64)
    r = b - O.spmv(rp, ci, v, x)
    assert np.linalg.norm(r) <= 1.01 * TOL * np.linalg.norm(b)


def test_gmres_uneven_magnitudes(ctx):
    """Right-hand side over 200 decades: the fixed-point sums align every term to the largest of its sum, so the
    residual reached is the one a 64-bit sum reports."""
    rp, ci, v, b = banded(3000, 9)
    b = b * 10.0 ** np.random.default_rng(1).uniform(-200, 0, b.size)
    _, x = solve(ctx, (rp, ci, v), b, 50, 0, tf.PREC_FP64)
    r = b - O.spmv(rp, ci, v, x)
    assert np.linalg.norm(r) <= 1.01 * TOL * np.linalg.norm(b)


def test_mixed_iterations_near_the_attainable_residual(ctx):
    """Cahn-Hilliard steps on a 30^3 torus to 1e-13: the restarts' basis vectors change length a thousandfold between
    two steps, and the mixed solver needs about the FP64 solver's iterations only while every norm keeps its bits
    (with norms in fixed units it took 14,000 instead of 800)."""
    n = 30
    its = {}
    for prec in (tf.PREC_FP64, tf.PREC_MIXED):
        ctx.brick_cube(n, 1.6)
        ctx.levelset_analytic(tf.LS_TORUS, [1.0013, 0.4019, 2], False)
        _, m = ctx.distribute_dofs(tf.P1IF)
        ctx.setup_fe_system([tf.FORM_M, tf.FORM_A, tf.FORM_CN])
        x0 = np.concatenate([0.5 + np.random.default_rng(5).uniform(-0.01, 0.01, m), np.zeros(m)])
        ctx.vec_upload(tf.VEC_X, x0)
        st, it, res, _ = ctx.ch_steps_learned(3, 1e-3, 1.0, 0.02, 0.0, 1.0, 3.2 / n, tol=1e-13, precision=prec, learned=0)
        assert st == tf.OK and res.max() <= 1e-13
        its[prec] = it
    print(its)
    assert its[tf.PREC_MIXED].sum() <= 1.25 * its[tf.PREC_FP64].sum()


@pytest.mark.parametrize("precision", [tf.PREC_FP64, tf.PREC_MIXED])
def test_uneven_rows_beyond_the_cached_part_of_the_matrix(precision):
    """Blocks whose share of the matrix is several times the mean keep only its head in shared memory."""
    from tests.test_gpu_pcg_cluster import mul, spd

    m = 12000
    A = spd(m, lambda i: 30 if i < m // 10 else 0, seed=11)
    b = A[3]
    with tf.TraceFEM(0) as ctx:
        ctx.matrix_upload(*A[:3])
        ctx.vec_upload(tf.VEC_B, b)
        ctx.vec_upload(tf.VEC_X, np.zeros(m))
        st, it, res = ctx.gmres_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, restart=50, tol=1e-10, precision=precision)
        assert st == tf.OK and res <= 1e-10
        r = b - mul(A, ctx.vec_download(tf.VEC_X))
    # the FP64 solver stops on the rotated residual, which follows the true one of a well conditioned system closely
    assert np.linalg.norm(r) <= 1.01e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("limit", [0, 1, 5, 23])
@pytest.mark.parametrize("method,prec", [(0, tf.PREC_FP64), (1, tf.PREC_FP64), (0, tf.PREC_MIXED)])
def test_iteration_limit(ctx, limit, method, prec):
    """No step, fewer than a restart cycle and more: not converged, the steps counted, the residual that of x."""
    rp, ci, v, b = banded(700, 2)
    ctx.matrix_upload(rp, ci, v)
    ctx.vec_upload(tf.VEC_B, b)
    ctx.vec_upload(tf.VEC_X, np.zeros(b.size))
    st, it, res = ctx.gmres_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, restart=8, tol=0.0, max_iter=limit, method=method,
                                   precision=prec)
    assert st == tf.ERR_NOT_CONVERGED and it == limit
    r = b - O.spmv(rp, ci, v, ctx.vec_download(tf.VEC_X))  # D = 2 drops out of |D^-1 r| / |D^-1 b|
    want = np.linalg.norm(r) / np.linalg.norm(b)
    assert abs(res - want) <= 1e-6 * want + 1e-15
    # a start that solves the system needs no step
    ctx.vec_upload(tf.VEC_B, np.zeros(b.size))
    ctx.vec_upload(tf.VEC_X, np.zeros(b.size))
    st, it, res = ctx.gmres_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, restart=8, tol=1e-9, max_iter=limit, method=method,
                                   precision=prec)
    assert st == tf.OK and it == 0 and res == 0.0
