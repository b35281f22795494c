"""Resident FP64 PCG and the packed grid reductions: sizes around slices and block shares, jumps of the summed values."""
import numpy as np
import pytest

import drops_gb300 as tf
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from drops_gb300 import build

    build.build()
    c = tf.TraceFEM()
    yield c
    c.close()


def spd(m, seed, decades=0.0):
    """Symmetric CSR matrix S B S with B's diagonal 2 and off-diagonal row sums of absolute values at most 1.5 (so
    0.5 <= B <= 3.5), S diagonal over `decades` decades."""
    rng = np.random.default_rng(seed)
    d = np.unique([1, 5, max(m // 4, 1)])
    rows, cols, vals = [np.arange(m)], [np.arange(m)], [np.full(m, 2.0)]
    for k in d:
        i = np.arange(max(m - k, 0))
        w = rng.uniform(-1.0, 1.0, i.size) * 0.25
        rows += [i, i + k]
        cols += [i + k, i]
        vals += [w, w]
    rows, cols, vals = (np.concatenate(x) for x in (rows, cols, vals))
    o = np.lexsort((cols, rows))
    s = 10.0 ** rng.uniform(-decades / 2, decades / 2, m)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int64)
    return rp, cols[o].astype(np.int64), (vals * s[rows] * s[cols])[o], rng.standard_normal(m), s


@pytest.mark.parametrize("m", [1, 31, 33, 512, 513, 4097, 20011, 200003])
@pytest.mark.parametrize("precision", [tf.PREC_FP64, tf.PREC_MIXED])
def test_pcg_sizes(ctx, m, precision):
    """Every size from one row to runs beyond the blocks' shared memory.  Both solutions have |r| <= tol |b| and
    |B^-1|_2 <= 2, so they differ by at most 4 tol |b| (10% more for the rounding of the residuals)."""
    tol = 1e-10
    rp, ci, v, b, _ = spd(m, m)
    ctx.matrix_upload(rp, ci, v)
    ctx.vec_upload(tf.VEC_B, b)
    ctx.vec_upload(tf.VEC_X, np.zeros(m))
    st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=tol, precision=precision)
    x = ctx.vec_download(tf.VEC_X)
    _, ox, oit, _ = O.pcg_jacobi(rp, ci, v, b, tol=tol)
    assert st == tf.OK and res <= tol
    assert np.linalg.norm(x - ox) <= 4.4 * tol * np.linalg.norm(b)
    if precision == tf.PREC_FP64:
        assert abs(it - oit) <= 1, (it, oit)


@pytest.mark.parametrize("decades", [6, 12])
def test_pcg_jumping_residuals(ctx, decades):
    """Rows scaled over many decades: Jacobi-PCG is that of the unscaled matrix, but <r, r> falls and rises by orders
    of magnitude from one iteration to the next, past the range of a packed sum's unit, and the reduction is repeated
    in floating point.  Iterations as the oracle's; residual checked in 64 bits."""
    tol = 1e-9
    rp, ci, v, b, s = spd(3000, 5, decades)
    b = b * s
    ctx.matrix_upload(rp, ci, v)
    ctx.vec_upload(tf.VEC_B, b)
    ctx.vec_upload(tf.VEC_X, np.zeros(b.size))
    st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=tol)
    x = ctx.vec_download(tf.VEC_X)
    _, ox, oit, _ = O.pcg_jacobi(rp, ci, v, b, tol=tol)
    assert st == tf.OK and abs(it - oit) <= 1, (it, oit)
    assert np.linalg.norm(b - O.spmv(rp, ci, v, x)) <= 1.01 * tol * np.linalg.norm(b)


def test_pcg_zero_and_converged_start(ctx):
    """b = 0 (every sum zero) and a start that already solves the system: no iteration, x unchanged."""
    rp, ci, v, b, _ = spd(1000, 7)
    ctx.matrix_upload(rp, ci, v)
    ctx.vec_upload(tf.VEC_B, np.zeros(1000))
    ctx.vec_upload(tf.VEC_X, np.zeros(1000))
    st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=1e-10)
    assert st == tf.OK and it == 0 and not ctx.vec_download(tf.VEC_X).any()
    ctx.vec_upload(tf.VEC_X, b)
    ctx.vec_upload(tf.VEC_B, O.spmv(rp, ci, v, b))
    st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=1e-10)
    assert st == tf.OK and it == 0 and np.array_equal(ctx.vec_download(tf.VEC_X), b)


@pytest.mark.parametrize("m,extra", [(400000, 0), (60000, 80)])
def test_systems_beyond_shared_memory_build_no_plan(monkeypatch, m, extra):
    """Too many rows, or too many entries, for the blocks' shared memory: the first solve launches what it launches with
    the resident solver off."""
    rng = np.random.default_rng(2)
    if extra:  # a band: the 16-bit columns of a block (60000 * 321 * 2 / 152 bytes) exceed its 227 KB
        off = np.arange(-extra * 2, extra * 2 + 1)
    else:
        off = np.arange(-1, 2)
    cols = np.arange(m)[:, None] + off[None, :]
    keep = (cols >= 0) & (cols < m)
    vals = np.where(off == 0, 2.0 * len(off), -1.0) * np.ones((m, 1))
    rp = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int64)
    b = rng.standard_normal(m)
    launches = []
    for resident in ("0", "1"):
        monkeypatch.setenv("TF_PCG_RESIDENT", resident)
        with tf.TraceFEM(0) as ctx:
            ctx.matrix_upload(rp, cols[keep].astype(np.int64), vals[keep])
            ctx.vec_upload(tf.VEC_B, b)
            ctx.vec_upload(tf.VEC_X, np.zeros(m))
            n0 = ctx.launch_count()
            st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=1e-10)
            launches.append(ctx.launch_count() - n0)
            assert st == tf.OK and res <= 1e-10
    assert launches[0] == launches[1]
