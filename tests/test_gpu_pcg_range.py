"""Stopping test and scalars of the FP64 PCG outside the ordinary range: tolerances below zero, right-hand sides whose
squares leave the doubles' normal range."""
import numpy as np
import pytest

import drops_gb300 as tf
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

M = 2000  # nodes of a chain, shuffled


def system():
    rng = np.random.default_rng(11)
    p = rng.permutation(M)
    rows, cols, vals = [p], [p], [rng.uniform(2.01, 2.5, M)]
    for a, b in ((p[:-1], p[1:]), (p[1:], p[:-1])):
        rows, cols, vals = rows + [a], cols + [b], vals + [np.full(M - 1, -1.0)]
    rows, cols, vals = (np.concatenate(x) for x in (rows, cols, vals))
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=M))]).astype(np.int64)
    return rp, cols[o].astype(np.int64), vals[o], rng.standard_normal(M)


@pytest.fixture(params=["8", "0"], ids=["cluster", "grid"])
def ctx(request, monkeypatch):
    monkeypatch.setenv("TF_PCG_CLUSTER", request.param)
    with tf.TraceFEM(0) as c:
        c.matrix_upload(*system()[:3])
        yield c


def solve(ctx, b, **kw):
    ctx.vec_upload(tf.VEC_B, b)
    ctx.vec_upload(tf.VEC_X, np.zeros(M))
    return ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, **kw)


@pytest.mark.parametrize("precision", [tf.PREC_FP64, tf.PREC_MIXED])
@pytest.mark.parametrize("rel", [True, False])
def test_negative_tolerance_is_never_reached(ctx, precision, rel):
    b = system()[3]
    st, it, res = solve(ctx, b, tol=-0.9, max_iter=7, rel=rel, precision=precision)
    assert st == tf.ERR_NOT_CONVERGED and it == 7
    r = b - O.spmv(*system()[:3], ctx.vec_download(tf.VEC_X))
    want = np.linalg.norm(r) / (np.linalg.norm(b) if rel else 1.0)
    assert abs(res - want) <= 1e-6 * want


def test_overflowing_norm_is_not_converged(ctx):
    """|b|^2 overflows: the residual over |b| is no number, so no tolerance is reached."""
    st, it, res = solve(ctx, system()[3] * 2.0**600, tol=1e-10, max_iter=5)
    assert st == tf.ERR_NOT_CONVERGED and it == 5


@pytest.mark.parametrize("power", [-486, -400, 400, 480])
def test_scaled_right_hand_side(ctx, power):
    """b times a power of two: the iterates scale along.  Where the squares of the last residuals are subnormal (2^-486:
    <r, r> ends near 2^-1030, with some 44 bits left) the count may move by one."""
    rp, ci, v, b = system()
    _, it, _ = solve(ctx, b, tol=1e-10)
    x = ctx.vec_download(tf.VEC_X)
    st, jt, res = solve(ctx, b * 2.0**power, tol=1e-10, max_iter=4 * it)
    y = ctx.vec_download(tf.VEC_X) * 2.0**-power
    assert st == tf.OK and res <= 1e-10 and abs(jt - it) <= (1 if power == -486 else 0)
    # both residuals are at most 1e-10 |b|, the smallest eigenvalue is at least 0.01
    assert np.linalg.norm(x - y) <= 2e-8 * np.linalg.norm(b)
