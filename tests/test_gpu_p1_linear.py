"""P1 forms on tets with a linear level set (closed forms, facet lists), beside the FP64 kernel on the same problem."""

import numpy as np
import pytest

import drops_gb300 as tf
from helpers import mat_close

pytestmark = pytest.mark.gpu

FORMS = [tf.FORM_M, tf.FORM_A, tf.FORM_CN]
LOADS = [(tf.RHS_CONST, [2.5]), (tf.RHS_SPHERE_XYZ, [0.0, 0.1, -0.05, 1.0, 13.0]), (tf.RHS_NONE, [])]


@pytest.fixture(scope="module")
def ctx():
    with tf.TraceFEM(0) as c:
        yield c


def forms(ctx, kernel, rhs, par):
    ctx.assemble_options(kernel)
    try:
        ctx.setup_fe_system(FORMS, rhs, par)
    finally:
        ctx.assemble_options(tf.ASM_KERNEL_PAIR)
    rp = ctx.matrix(tf.FORM_M)[0]
    return rp, [ctx.matrix(f)[2] for f in FORMS] + ([ctx.vec_download(tf.VEC_RHS)] if rhs != tf.RHS_NONE else [])


def compare(ctx, exact=None):
    # the parity bound of the pair kernels, 1e-12 of the row's scale
    for rhs, par in LOADS:
        rp, a = forms(ctx, tf.ASM_KERNEL_PAIR, rhs, par)
        _, b = forms(ctx, tf.ASM_KERNEL_FP64, rhs, par)
        if exact is not None:
            b[0], b[1] = exact[0], exact[1]
            if rhs == tf.RHS_CONST:
                b[3] = par[0] * exact[2]
        for k, (x, y) in enumerate(zip(a, b)):
            assert np.all(np.isfinite(x))
            ok, err = mat_close(x, y, rp if k < 3 else None)
            assert ok, (rhs, k, err)


def exact_forms(ctx, n, a):
    """M, A and the load of f = 1 from the planar cuts in extended precision (no node value may be 0).  The FP64 kernel
    forms areas from differences of world coordinates, which costs it up to 1.2e-12 of a row's scale where the cuts are
    tiny."""
    L = np.longdouble
    rp, ci, _ = ctx.matrix(tf.FORM_M)
    lv, _ = ctx.levelset_download()
    dof = ctx.dofs()[0]
    off = np.zeros((6, 4, 3), np.int64)
    for t, (p, q) in enumerate([(2, 1), (2, 0), (1, 2), (1, 0), (0, 2), (0, 1)]):
        off[t, 1, p] = off[t, 2, p] = off[t, 2, q] = 1
        off[t, 3] = 1
    cube = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 1, 1, 3)
    P = (cube + off).reshape(-1, 4, 3)
    T = (P[..., 0] * (n + 1) + P[..., 1]) * (n + 1) + P[..., 2]
    sg = lv[T] > 0
    cut = sg.any(1) & ~sg.all(1)
    T, P, sg = T[cut], P[cut], sg[cut]
    f = lv[T].astype(L)
    X = (-a + P[..., ::-1] * (2 * a / n)).astype(L)
    E = X[:, 1:] - X[:, :1]
    G = np.zeros(X.shape, L)
    for k in range(3):
        G[:, k + 1] = np.cross(E[:, (k + 1) % 3], E[:, (k + 2) % 3])
    G /= (E[:, 0] * G[:, 1]).sum(1)[:, None, None]
    G[:, 0] = -G[:, 1:].sum(1)
    nr = (f[:, :, None] * G).sum(1)
    nr /= np.sqrt((nr**2).sum(1))[:, None]
    S = G - (G * nr[:, None]).sum(2)[:, :, None] * nr[:, None]
    area, M, F = np.zeros(len(T), L), np.zeros((len(T), 4, 4), L), np.zeros((len(T), 4), L)
    code = (sg * np.array([1, 2, 4, 8])).sum(1)
    for mask in range(1, 15):
        sel = np.nonzero(code == mask)[0]
        pts = []
        for i in (i for i in range(4) if mask >> i & 1):
            for j in (j for j in range(4) if not mask >> j & 1):
                B = np.zeros((len(sel), 4), L)
                B[:, j] = f[sel, i] / (f[sel, i] - f[sel, j])
                B[:, i] = 1 - B[:, j]
                pts.append(B)
        for tri in [(0, 1, 2)] if len(pts) == 3 else [(0, 1, 2), (1, 3, 2)]:
            B = np.stack([pts[k] for k in tri], 1)
            W = (B[:, :, :, None] * X[sel][:, None]).sum(2)
            ar = np.sqrt((np.cross(W[:, 1] - W[:, 0], W[:, 2] - W[:, 0]) ** 2).sum(1)) / 2
            mid = B.sum(1)
            area[sel] += ar
            F[sel] += ar[:, None] / 3 * mid
            M[sel] += ar[:, None, None] / 12 * ((B[:, :, :, None] * B[:, :, None, :]).sum(1) + mid[:, :, None] * mid[:, None, :])
    A = area[:, None, None] * (S[:, :, None] * S[:, None]).sum(3)
    m, D = len(rp) - 1, dof[T].astype(np.int64)
    keys = np.repeat(np.arange(m), np.diff(rp)) * m + ci
    at = np.searchsorted(keys, (D[:, :, None] * m + D[:, None, :]).ravel())
    out = []
    for K in (M, A):
        v = np.zeros(len(keys), L)
        np.add.at(v, at, K.ravel())
        out.append(v.astype(np.float64))
    v = np.zeros(m, L)
    np.add.at(v, D.ravel(), F.ravel())
    return out + [v.astype(np.float64)]


# one cube to past the sizes where the lanes per tet (4,864 cut tets) and the registers (58,368) change; odd counts
# leave a ragged last block
@pytest.mark.parametrize("n", [2, 3, 7, 16, 25, 26, 86, 88])
@pytest.mark.parametrize("kind,par", [(tf.LS_SPHERE, [0.0031, -0.0047, 0.0083, 1.0027]), (tf.LS_TORUS, [1.0, 0.4, 2])])
def test_linear_level_set(ctx, n, kind, par):
    ctx.brick_cube(n, 5.0 / 3.0)
    ctx.levelset_analytic(kind, par, False)
    na, _ = ctx.distribute_dofs(tf.P1IF)
    if na:
        ctx.setup_fe_system(FORMS)
        zero = (ctx.levelset_download()[0] == 0).any()
        compare(ctx, None if zero else exact_forms(ctx, n, 5.0 / 3.0))


def test_scales_of_the_level_set(ctx):
    """Cuts near and across the bricks' planes, and level sets so small or so large that the square of the gradient
    leaves the range in which the plane's normal gives the areas."""
    n, a = 6, 1.0
    ctx.brick_cube(n, a)
    g = np.linspace(-a, a, n + 1)
    z, y, x = np.meshgrid(g, g, g, indexing="ij")
    for lv in (x + 1e-3, x + y + 0.013, x + 0.9 * y + 0.8 * z + 0.01, x + 1e-3 * y + a / n):
        for scale in (1.0, 1e-8, 1e9):
            ctx.levelset_upload((lv * scale).ravel())
            na, _ = ctx.distribute_dofs(tf.P1IF)
            assert na > 0
            compare(ctx)
    # the normal overflows in the FP64 kernel too: the mass matrix and the load alone
    for scale in (1e-160, 1e160):
        ctx.levelset_upload(((x + 0.3 * y + 0.11) * scale).ravel())
        ctx.distribute_dofs(tf.P1IF)
        for rhs, par in LOADS[:2]:
            out = []
            for kernel in (tf.ASM_KERNEL_PAIR, tf.ASM_KERNEL_FP64):
                ctx.assemble_options(kernel)
                ctx.setup_fe_system([tf.FORM_M], rhs, par)
                ctx.assemble_options(tf.ASM_KERNEL_PAIR)
                out.append((ctx.matrix(tf.FORM_M), ctx.vec_download(tf.VEC_RHS)))
            ok, err = mat_close(out[0][0][2], out[1][0][2], out[0][0][0])
            assert ok, (scale, err)
            ok, err = mat_close(out[0][1], out[1][1])
            assert ok, (scale, err)


@pytest.mark.parametrize("n", [5, 24, 60])
@pytest.mark.parametrize("share", [0.02, 0.5, 0.98, 1.0])
def test_linear_and_other_tets_together(ctx, n, share):
    """Edge values off the mean on a share of the edges: those tets take the general kernels, in any mixture."""
    rng = np.random.default_rng(n)
    ctx.brick_cube(n, 5.0 / 3.0)
    ctx.levelset_analytic(tf.LS_SPHERE, [0.0, 0.1, 0.0, 1.0], False)
    lv, le = ctx.levelset_download()
    le = np.where(rng.uniform(size=le.size) < share, le + 1e-3 / n * rng.uniform(-1.0, 1.0, le.size), le)
    ctx.levelset_upload(lv, le)
    ctx.distribute_dofs(tf.P1IF)
    compare(ctx)


@pytest.mark.parametrize("rhs,par", LOADS)
def test_repeated_calls_agree(ctx, rhs, par):
    """The tets that are not linear are listed in the order in which warps reach the list, which differs from call to
    call; every tet writes its own record, so the results are the same bits."""
    rng = np.random.default_rng(8)
    ctx.brick_cube(40, 5.0 / 3.0)
    ctx.levelset_analytic(tf.LS_SPHERE, [0.0, 0.1, 0.0, 1.0], False)
    lv, le = ctx.levelset_download()
    ctx.levelset_upload(lv, np.where(rng.uniform(size=le.size) < 0.1, le + 2e-5 * rng.uniform(-1.0, 1.0, le.size), le))
    ctx.distribute_dofs(tf.P1IF)
    first = None
    for _ in range(8):
        now = [x.tobytes() for x in forms(ctx, tf.ASM_KERNEL_PAIR, rhs, par)[1]]
        assert first is None or now == first
        first = now
