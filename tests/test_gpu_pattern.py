"""Numbering and CSR pattern at the edges of their kernels: values without a plain sign bit, rows with many contributions."""
import numpy as np
import pytest

import drops_gb300 as tf
from oracle import pyoracle as O
from tests.helpers import MAT_RTOL, mat_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from drops_gb300 import build

    build.build()
    c = tf.TraceFEM()
    yield c
    c.close()


@pytest.mark.parametrize("n", [(1, 1, 1), (7, 1, 2), (5, 9, 12), (31, 17, 3)])
@pytest.mark.parametrize("p2", [False, True])
@pytest.mark.parametrize("dist", [0.0, 0.05, -1.0])
def test_classification_odd_values(ctx, n, p2, dist):
    """Level-set values whose high word does not tell the sign: subnormals, infinities, NaN, tiny normals.  Active
    tets and numbers as the oracle's, which evaluates distance() in FP64; narrow band and negative distance too."""
    om = O.brick(n, orig=np.array([-1.0, -1.0, -1.0]), e=np.diag([2.0, 2.0, 2.0]))
    rng = np.random.default_rng(sum(n) + p2)
    lv = om.coords @ np.array([0.3, -0.2, 0.5]) + 0.01 * rng.standard_normal(om.nv)
    le = 0.5 * (lv[om.edge_v[:, 0]] + lv[om.edge_v[:, 1]]) + 0.01 * rng.standard_normal(om.ne)
    odd = np.array([5e-324, -5e-324, 1e-310, -1e-310, np.inf, -np.inf, np.nan, 2.3e-308, -2.3e-308])
    for a in (lv, le):
        k = rng.integers(0, a.size, max(a.size // 12, 1))
        a[k] = odd[rng.integers(0, odd.size, k.size)]
    lv[lv == 0.0], le[le == 0.0] = 1e-300, 1e-300
    ctx.brick([-1, -1, -1], [2, 0, 0], [0, 2, 0], [0, 0, 2], *n)
    ctx.levelset_upload(lv, le)
    na, nd = ctx.distribute_dofs(tf.P2IF if p2 else tf.P1IF, dist)
    st, ona, ond, odv, ode, oact = O.distribute_dofs(om, lv, le, p2, dist)
    assert st == O.OK and (na, nd) == (ona, ond)
    dv, de, act, _ = ctx.dofs()
    assert np.array_equal(act, np.nonzero(oact)[0]) and np.array_equal(dv, odv)
    if p2:
        assert np.array_equal(de, ode)


def star(tris, pts):
    """Tets from the origin (vertex 0) to the triangles of a sphere, with an edge table."""
    tv = np.concatenate([np.zeros((len(tris), 1), int), np.asarray(tris) + 1], axis=1)
    ends = [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (2, 3)]
    e = np.stack([np.sort(tv[:, list(p)], axis=1) for p in ends], axis=1)
    ev, inv = np.unique(e.reshape(-1, 2), axis=0, return_inverse=True)
    coords = np.concatenate([np.zeros((1, 3)), pts])
    return O.Mesh(coords, tv.astype(np.int32), inv.reshape(-1, 6).astype(np.int32), ev.astype(np.int32))


def sphere_tris(levels):
    p = [np.array(x, float) for x in [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]]
    t = [(0, 2, 4), (2, 1, 4), (1, 3, 4), (3, 0, 4), (2, 0, 5), (1, 2, 5), (3, 1, 5), (0, 3, 5)]
    for _ in range(levels):
        mid, new = {}, []

        def m(a, b):
            k = (min(a, b), max(a, b))
            if k not in mid:
                mid[k] = len(p)
                x = p[a] + p[b]
                p.append(x / np.linalg.norm(x))
            return mid[k]

        for a, b, c in t:
            ab, bc, ca = m(a, b), m(b, c), m(c, a)
            new += [(a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca)]
        t = new
    return t, np.array(p)


@pytest.mark.parametrize("levels,p2", [(0, False), (0, True), (1, False), (1, True), (2, False)])
def test_rows_with_many_contributions(ctx, levels, p2):
    """The centre vertex of a star of 8, 32 or 128 cut tets: 32 to 512 contributions in its row (one to eight keys per
    lane, then shared memory).  Pattern bit-exact, values within the matrix tolerance."""
    om = star(*sphere_tris(levels))
    par = [0.02, -0.01, 0.015, 0.55]
    lv, le = O.levelset(om, O.LS_SPHERE, par, p2)
    ctx.mesh_upload(om.coords, om.tet_v, om.tet_e, om.edge_v)
    ctx.levelset_upload(lv, le)
    na, nd = ctx.distribute_dofs(tf.P2IF if p2 else tf.P1IF)
    st, ona, ond, odv, ode, oact = O.distribute_dofs(om, lv, le, p2)
    assert (na, nd) == (ona, ond)
    forms = [tf.FORM_M, tf.FORM_A, tf.FORM_CN]
    ctx.setup_fe_system(forms, tf.RHS_CONST, [1.0])
    opts = O.make_opts(p2, forms, O.RHS_CONST, [1.0])
    _, orp, oci, vals, rhs = O.assemble(om, lv, le, oact, odv, ode, ond, opts)
    for f in forms:
        rp, ci, v = ctx.matrix(f)
        assert np.array_equal(rp, orp) and np.array_equal(ci, oci)
        ok, err = mat_close(v, vals[f], orp)
        assert ok, (f, err)
    assert np.abs(ctx.vec_download(tf.VEC_RHS) - rhs).max() <= MAT_RTOL * np.abs(rhs).max()


def test_row_beyond_capacity(ctx):
    """128 P2 tets at one vertex: 1,280 contributions in a row, refused as before."""
    om = star(*sphere_tris(2))
    lv, le = O.levelset(om, O.LS_SPHERE, [0.02, -0.01, 0.015, 0.55], True)
    ctx.mesh_upload(om.coords, om.tet_v, om.tet_e, om.edge_v)
    ctx.levelset_upload(lv, le)
    ctx.distribute_dofs(tf.P2IF)
    with pytest.raises(tf.TraceFEMError) as e:
        ctx.setup_fe_system([tf.FORM_M])
    assert e.value.status == tf.ERR_CAPACITY
