"""PCG of one system per thread-block cluster: shares of every shape, all placements of the matrix, the batch."""

import numpy as np
import pytest

import drops_gb300 as tf
from drops_gb300.workloads import ellipsoid_batch

pytestmark = pytest.mark.gpu

TOL = 1e-10


def spd(m, extra, seed):
    """Diagonally dominant symmetric matrix: a chain plus extra(i) random links per row; CSR."""
    rng = np.random.default_rng(seed)
    a = {}
    for i in range(m):
        links = [i - 1] + list(rng.integers(0, m, extra(i)))
        for j in links:
            if 0 <= j < m and j != i:
                w = -rng.uniform(0.1, 1.0)
                a[(i, j)] = w
                a[(j, i)] = w
    keys = np.array(sorted(a), dtype=np.int64).reshape(-1, 2)
    vals = np.array([a[tuple(k)] for k in keys]) if len(keys) else np.zeros(0)
    diag = 0.05 + rng.uniform(0.0, 0.1, m)
    if len(keys):
        diag += np.bincount(keys[:, 0], -vals, m)
    rows = np.concatenate([keys[:, 0], np.arange(m)])
    cols = np.concatenate([keys[:, 1], np.arange(m)])
    vals = np.concatenate([vals, diag])
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int64)
    return rp, cols[o].astype(np.int64), vals[o], rng.standard_normal(m)


def mul(A, x):
    rp, ci, v, _ = A
    return np.add.reduceat(np.concatenate([v * x[ci], [0.0]]), rp[:-1])


def cg(A, tol):
    rp, ci, v, b = A
    m = len(b)
    d = np.array([v[rp[i]:rp[i + 1]][ci[rp[i]:rp[i + 1]] == i][0] for i in range(m)])
    x, r = np.zeros(m), b.copy()
    nb = np.linalg.norm(b)
    z = r / d
    p, rho, it = z.copy(), r @ z, 0
    while np.linalg.norm(r) > tol * nb:
        q = mul(A, p)
        al = rho / (p @ q)
        x += al * p
        r -= al * q
        z = r / d
        rho, old = r @ z, rho
        p = z + (rho / old) * p
        it += 1
    return it


@pytest.fixture
def context(monkeypatch):
    made = []

    def make(ctas):
        monkeypatch.setenv("TF_PCG_CLUSTER", str(ctas))
        made.append(tf.TraceFEM(0))
        return made[-1]

    yield make
    for c in made:
        c.close()


# (rows, links per row): one row, around a slice, ragged shares, a few long rows, more entries than the shared
# memory holds, and shares far above the even one (their last slices are read from the CSR arrays)
SYSTEMS = {
    "one": (1, lambda i: 0),
    "slice-1": (31, lambda i: 2),
    "slice+1": (33, lambda i: 2),
    "ragged": (519, lambda i: i % 7),
    "long rows": (700, lambda i: 300 if i in (5, 650) else 1),
    "beyond shared memory": (3100, lambda i: 16),
    "uneven shares": (4000, lambda i: 40 if i < 400 else 0),
}
_cache = {}


def system(name):
    if name not in _cache:
        A = spd(*SYSTEMS[name], seed=7)
        _cache[name] = A, cg(A, TOL)
    return _cache[name]


@pytest.mark.parametrize("ctas", [1, 2, 4, 8])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_single_system(context, name, ctas):
    A, its = system(name)
    b = A[3]
    ctx = context(ctas)
    ctx.matrix_upload(*A[:3])
    ctx.vec_upload(tf.VEC_B, b)
    for precision in (tf.PREC_FP64, tf.PREC_MIXED):
        ctx.vec_upload(tf.VEC_X, np.zeros(len(b)))
        n0 = ctx.launch_count()
        st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=TOL, precision=precision)
        assert st == tf.OK and res <= TOL
        assert ctx.launch_count() == n0 + 1  # the cluster kernel, no layout
        # the recursive FP64 residual of a system this well conditioned follows the true one to a few ulps of |b|
        assert np.linalg.norm(b - mul(A, ctx.vec_download(tf.VEC_X))) <= 1.01 * TOL * np.linalg.norm(b)
        assert abs(it - its) <= (1 if precision == tf.PREC_FP64 else 2 + its // 4)


def test_iteration_limit_and_start_value(context):
    A, its = system("ragged")
    b = A[3]
    ctx = context(4)
    ctx.matrix_upload(*A[:3])
    ctx.vec_upload(tf.VEC_B, b)
    for precision in (tf.PREC_FP64, tf.PREC_MIXED):
        for limit in (0, 3):
            ctx.vec_upload(tf.VEC_X, np.zeros(len(b)))
            st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=TOL, max_iter=limit, precision=precision,
                                         check=False)
            assert st == tf.ERR_NOT_CONVERGED and it == limit
            r = np.linalg.norm(b - mul(A, ctx.vec_download(tf.VEC_X))) / np.linalg.norm(b)
            assert abs(res - r) <= 1e-6 * r
        ctx.vec_upload(tf.VEC_X, np.zeros(len(b)))
        ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=TOL, precision=precision)
        st, it, _ = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=2 * TOL, precision=precision)
        assert st == tf.OK and it == 0


def test_first_and_later_solves_on_a_pattern_agree(monkeypatch):
    """By rule the first solve of a small system takes a cluster, the next the grid-wide kernels."""
    monkeypatch.delenv("TF_PCG_CLUSTER", raising=False)
    A, its = system("ragged")
    b = A[3]
    with tf.TraceFEM(0) as ctx:
        ctx.matrix_upload(*A[:3])
        ctx.vec_upload(tf.VEC_B, b)
        xs = []
        for _ in range(3):
            ctx.vec_upload(tf.VEC_X, np.zeros(len(b)))
            st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=TOL)
            assert st == tf.OK and abs(it - its) <= 1
            xs.append(ctx.vec_download(tf.VEC_X))
        # both stop at a residual of TOL |b|; the smallest eigenvalue is at least 0.05
        for x in xs[1:]:
            assert np.linalg.norm(x - xs[0]) <= 2 * TOL * np.linalg.norm(b) / 0.05


@pytest.mark.parametrize("ctas", [1, 2, 4, 8])
@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("precision", [tf.PREC_MIXED, tf.PREC_FP64])
def test_batch(context, ctas, graph, precision):
    """Uneven ellipsoids: every instance reaches the tolerance, and agrees with the CTA-per-problem kernel."""
    W = ellipsoid_batch(40, nmin=6, nmax=30, seed=99)
    forms = [tf.FORM_M, tf.FORM_A, tf.FORM_CN]

    def solve(ctx, lanes):
        ctx.brick_batch(W["n"], W["orig"], W["axes"])
        ctx.levelset_analytic_batch(tf.LS_ELLIPSOID, W["par"], p2=False)
        _, m = ctx.distribute_dofs(tf.P1IF)
        ctx.setup_fe_system(forms, tf.RHS_SPHERE_XYZ, [0.0, 0.0, 0.0, 1.0, 12.0])
        ctx.batch_lincomb(forms, np.stack([np.ones(40), np.ones(40), W["h"]], axis=1))
        ctx.batch_config(lanes, 256 if lanes else 0, use_graph=graph)
        out = []
        for _ in range(2):
            ctx.vec_fill(tf.VEC_X, m, 0.0)
            st, it, res = ctx.batch_pcg_jacobi(tf.MAT_SYS, tf.VEC_RHS, tf.VEC_X, tol=TOL, precision=precision)
            assert st == tf.OK and res.max() <= TOL
            out.append(ctx.vec_download(tf.VEC_X))
        assert np.array_equal(out[0], out[1])
        return out[0], it

    ctx = context(ctas)
    x, it = solve(ctx, 0)
    rp, ci, v = ctx.matrix(tf.MAT_SYS)
    b = ctx.vec_download(tf.VEC_RHS)
    rows = ctx.batch_info(nnz=False)[2]
    r = b - mul((rp, ci, v, b), x)
    for i in range(40):
        s = slice(rows[i], rows[i + 1])
        assert np.linalg.norm(r[s]) <= 1.01 * TOL * np.linalg.norm(b[s])
    y, jt = solve(ctx, 4)
    # both within TOL of the solution in the residual; the systems' condition numbers are below 1e4
    for i in range(40):
        s = slice(rows[i], rows[i + 1])
        assert np.linalg.norm(x[s] - y[s]) <= 2e4 * TOL * np.linalg.norm(y[s])
    assert np.all(np.abs(it - jt) <= (1 if precision == tf.PREC_FP64 else 2 + jt // 4))


@pytest.mark.parametrize("precision", [tf.PREC_MIXED, tf.PREC_FP64])
def test_batch_uploaded_matrix(context, precision):
    """A caller's matrix as large as the numbering: block diagonal it is solved like the assembled one; with entries
    between instances, which no cluster can hold, the call ends within its iterations and the context stays usable."""
    W = ellipsoid_batch(9, nmin=6, nmax=20, seed=5)
    forms = [tf.FORM_M, tf.FORM_A, tf.FORM_CN]
    ctx = context(8)
    ctx.brick_batch(W["n"], W["orig"], W["axes"])
    ctx.levelset_analytic_batch(tf.LS_ELLIPSOID, W["par"], p2=False)
    _, m = ctx.distribute_dofs(tf.P1IF)
    ctx.setup_fe_system(forms, tf.RHS_SPHERE_XYZ, [0.0, 0.0, 0.0, 1.0, 12.0])
    ctx.batch_lincomb(forms, np.stack([np.ones(9), np.ones(9), W["h"]], axis=1))
    rp, ci, v = ctx.matrix(tf.MAT_SYS)
    b = ctx.vec_download(tf.VEC_RHS)
    rows = ctx.batch_info(nnz=False)[2]

    def solve(mat, **kw):
        ctx.vec_fill(tf.VEC_X, m, 0.0)
        st, it, res = ctx.batch_pcg_jacobi(mat, tf.VEC_RHS, tf.VEC_X, tol=TOL, precision=precision, check=False, **kw)
        return st, res, ctx.vec_download(tf.VEC_X)

    def solved(st, res, x):
        r = b - mul((rp, ci, v, b), x)
        return st == tf.OK and res.max() <= TOL and all(
            np.linalg.norm(r[s:e]) <= 1.01 * TOL * np.linalg.norm(b[s:e]) for s, e in zip(rows[:-1], rows[1:]))

    ctx.matrix_upload(rp, ci, v)
    assert solved(*solve(tf.MAT_USER))
    # the last row of every instance linked to the first and the last of all others
    ends = np.unique(np.concatenate([rows[:-1], rows[1:] - 1]))
    import scipy.sparse as sp

    E = sp.coo_matrix((np.full(len(ends) * (len(ends) - 1), -1e-3),
                       (np.repeat(ends, len(ends) - 1), np.concatenate([np.delete(ends, i) for i in range(len(ends))]))),
                      shape=(m, m))
    L = (sp.csr_matrix((v, ci, rp), shape=(m, m)) + E).tocsr()
    L.sort_indices()
    ctx.matrix_upload(L.indptr.astype(np.int64), L.indices.astype(np.int64), L.data)
    assert solve(tf.MAT_USER, max_iter=40)[0] in (tf.OK, tf.ERR_NOT_CONVERGED)
    assert solved(*solve(tf.MAT_SYS))


def _no_memory(monkeypatch):
    monkeypatch.setenv("TF_PCG_CLUSTER_EXTRA_MB", str(1 << 30))  # more than any device has: the scratch cannot be had


@pytest.mark.parametrize("precision", [tf.PREC_FP64, tf.PREC_MIXED])
def test_single_system_without_room_for_a_cluster(context, monkeypatch, precision):
    """No memory for the cluster's scratch: the grid-wide kernels solve, and no error is left behind."""
    _no_memory(monkeypatch)
    A, its = system("ragged")
    b = A[3]
    ctx = context(4)
    ctx.matrix_upload(*A[:3])
    ctx.vec_upload(tf.VEC_B, b)
    ctx.vec_upload(tf.VEC_X, np.zeros(len(b)))
    st, it, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=TOL, precision=precision)
    assert st == tf.OK and res <= TOL
    assert np.linalg.norm(b - mul(A, ctx.vec_download(tf.VEC_X))) <= 1.01 * TOL * np.linalg.norm(b)
    assert abs(it - its) <= (1 if precision == tf.PREC_FP64 else 2 + its // 4)


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("precision", [tf.PREC_FP64, tf.PREC_MIXED])
@pytest.mark.parametrize("why", ["no memory", "rows"])
def test_batch_without_room_for_clusters(context, monkeypatch, precision, graph, why):
    """Scratch that cannot be had, and an instance of more rows than a cluster holds: a CTA per instance solves."""
    W = ellipsoid_batch(6, nmin=6, nmax=20, seed=31)
    if why == "rows":
        W["n"][2] = 160  # about 47,000 rows
    else:
        _no_memory(monkeypatch)
    forms = [tf.FORM_M, tf.FORM_A, tf.FORM_CN]
    ctx = context(8)
    ctx.brick_batch(W["n"], W["orig"], W["axes"])
    ctx.levelset_analytic_batch(tf.LS_ELLIPSOID, W["par"], p2=False)
    _, m = ctx.distribute_dofs(tf.P1IF)
    ctx.setup_fe_system(forms, tf.RHS_SPHERE_XYZ, [0.0, 0.0, 0.0, 1.0, 12.0])
    ctx.batch_lincomb(forms, np.stack([np.ones(6), np.ones(6), W["h"]], axis=1))
    rows = ctx.batch_info(nnz=False)[2]
    if why == "rows":
        assert rows[3] - rows[2] > 37000
    ctx.batch_config(0, 0, use_graph=graph)
    rp, ci, v = ctx.matrix(tf.MAT_SYS)
    b = ctx.vec_download(tf.VEC_RHS)
    for _ in range(2):
        ctx.vec_fill(tf.VEC_X, m, 0.0)
        st, it, res = ctx.batch_pcg_jacobi(tf.MAT_SYS, tf.VEC_RHS, tf.VEC_X, tol=TOL, precision=precision)
        assert st == tf.OK and res.max() <= TOL
        r = b - mul((rp, ci, v, b), ctx.vec_download(tf.VEC_X))
        for s, e in zip(rows[:-1], rows[1:]):
            assert np.linalg.norm(r[s:e]) <= 1.01 * TOL * np.linalg.norm(b[s:e])
