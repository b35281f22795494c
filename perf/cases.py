"""Timing cases of the TraceFEM path: what a program has the library do, through its public entry points.

A case is a dict of plain values; `prepare` makes what the program holds before the call (a context with its mesh
and level set, host arrays), `run` makes one pass and returns the pass's results, `work` states the bytes and
operations a pass cannot do without, and `exact` the results in 64-bit arithmetic where plain torch or numpy gives
them.  Kinds:

  step    one surface problem from the level set to the solution: DOF numbering, forms and load vector, linear
          combination, Jacobi-PCG to a relative residual of 1e-10, solution read back
  forms   the assembly call alone: numbering, forms and load vector, system matrix and load vector to the host
  batch   many uneven ellipsoid problems as one
  ch      time steps of the Cahn-Hilliard system on a torus
  refine  the brick refined towards the surface, then the P2 problem on the refined mesh
  quaqua  the isoparametric P2 forms on a fixed numbering
  spmv    one matrix-vector product of a program's own iteration
  user    a program's own CSR matrix handed to a solver with host vectors (the drop-in Solve call)
  noalloc the allocation-free PCG on device arrays of the caller
"""
import ctypes as C
import math

import numpy as np
import torch

import drops_gb300 as tf
from drops_gb300.workloads import BOX, ellipsoid_batch

TOL = 1e-10
FORMS = [tf.FORM_M, tf.FORM_A, tf.FORM_CN]
CH_BOX = 1.6
# The Cahn-Hilliard states depend on the solves a thousand times more than their residuals show (rows of vertices that
# hardly touch the surface): at 1e-13 they are settled to about ten digits.
CH_TOL = 1e-13


def listed():
    return [
        # the smallest problem people start with: the 16^3 P1 sphere, all in 64 bits; launches and host waits count
        dict(name="step_p1_16", kind="step", fe="p1", shape="sphere", n=16, prec="fp64", upload=False),
        # the headline problem: P2 sphere on 96^3 cubes, mixed precision
        dict(name="step_p2_96", kind="step", fe="p2", shape="sphere", n=96, prec="mixed", upload=False),
        # an odd-sized P2 torus with the solver's default precision
        dict(name="step_p2_41_torus", kind="step", fe="p2", shape="torus", n=41, prec="fp64", upload=False),
        # a step of a moving surface: new level-set values come from the host each pass
        dict(name="step_p1_61_upload", kind="step", fe="p1", shape="torus", n=61, prec="mixed", upload=True),
        # the drop-in assembly call on a large P1 torus, matrix and load vector wanted on the host
        dict(name="forms_p1_128", kind="forms", fe="p1", shape="torus", n=128),
        # 256 uneven ellipsoids, 16^3 to 64^3 cubes, as one batch
        dict(name="batch_256", kind="batch", count=256, nmin=16, nmax=64, prec="mixed"),
        # Cahn-Hilliard on the 128^3 torus, mixed precision with the learned warm start
        dict(name="ch_128_learned", kind="ch", n=128, steps=5, prec="mixed", learned=1),
        # the default Cahn-Hilliard loop (64 bits, modified Gram-Schmidt) on a small torus
        dict(name="ch_40_fp64", kind="ch", n=40, steps=2, prec="fp64", learned=-1),
        # the surface driver's mesh step and the P2 problem on the refined mesh
        dict(name="refine_p2_32", kind="refine", n=32, levels=2, width=0.05),
        # isoparametric P2 forms of the surfactant driver
        dict(name="quaqua_96", kind="quaqua", n=96),
        # one product with a P2 system matrix larger than L2
        dict(name="spmv_p2_192", kind="spmv", fe="p2", n=192),
        # a nonsymmetric system of the caller's through GMRES, ragged grid
        dict(name="user_gmres", kind="user", solver="gmres", method=0, k1=41, k2=37, k3=43),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)) - 1e-9)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "forms", "batch", "ch", "refine", "quaqua", "spmv", "user", "noalloc"])
    if kind == "step":
        fe, prec = rng.choice(["p1", "p2"]), rng.choice(["fp64", "mixed"])
        n = _log(rng, 10, 128 if fe == "p1" else 96 if prec == "mixed" else 72)
        return dict(kind=kind, fe=fe, shape=rng.choice(["sphere", "torus"]), n=n, prec=prec, upload=rng.random() < 0.3)
    if kind == "forms":
        fe = rng.choice(["p1", "p2"])
        return dict(kind=kind, fe=fe, shape=rng.choice(["sphere", "torus"]), n=_log(rng, 10, 128 if fe == "p1" else 64))
    if kind == "batch":
        nmin = _log(rng, 8, 24)
        return dict(kind=kind, count=_log(rng, 16, 200), nmin=nmin, nmax=rng.randint(nmin + 4, 60),
                    prec=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "ch":
        if rng.random() < 0.5:
            return dict(kind=kind, n=_log(rng, 16, 112), steps=rng.randint(2, 5), prec="mixed", learned=rng.choice([0, 1, 3]))
        return dict(kind=kind, n=_log(rng, 16, 48), steps=rng.randint(1, 2), prec="fp64", learned=rng.choice([-1, 0]))
    if kind == "refine":
        return dict(kind=kind, n=_log(rng, 8, 32), levels=rng.randint(1, 2), width=round(rng.uniform(0.02, 0.05), 4))
    if kind == "quaqua":
        return dict(kind=kind, n=_log(rng, 12, 96))
    if kind == "spmv":
        fe = rng.choice(["p1", "p2"])
        return dict(kind=kind, fe=fe, n=_log(rng, 16, 192))
    k = [_log(rng, 8, 62) for _ in range(3)]
    if kind == "noalloc":
        return dict(kind=kind, k1=k[0], k2=k[1], k3=k[2])
    solver = rng.choice(["gmres", "pcg", "pcg_mixed"])
    return dict(kind=kind, solver=solver, method=rng.randint(0, 1) if solver == "gmres" else 0, k1=k[0], k2=k[1], k3=k[2])


# ---------------------------------------------------------------------------------------------------------------
class State:
    """What the program keeps between calls; closes the context and frees its page-locked inputs when dropped."""

    def __init__(self, case):
        self.case, self.ctx, self.pinned = case, None, []

    def pin(self, data):
        a = tf.PinnedArray(data.size)
        self.pinned.append(a)
        a.array[:] = data
        return a.array

    def __del__(self):
        try:
            if self.ctx is not None:
                self.ctx.close()
            for a in self.pinned:
                a.free()
        except Exception:
            pass


def _surface(shape):
    """(half-width of the cube, level-set kind, parameters), a little off the round numbers whose level sets are exactly
    zero at nodes of some bricks."""
    if shape == "sphere":
        return BOX, tf.LS_SPHERE, [0.0031, -0.0047, 0.0083, 1.0027]
    return CH_BOX, tf.LS_TORUS, [1.0013, 0.4019, 2]


# directions (d3, d2, d1) of the edge classes in the library's numbering, each numbered by its lower vertex
_EDGE_DIRS = [(0, 0, 1), (0, 1, 0), (1, 0, 0), (0, 1, 1), (1, 0, 1), (1, 1, 0), (1, 1, 1)]


def _bend(n, wave, phase, p2):
    """A smooth positive factor at the vertices and edge midpoints of the n^3 brick.  A level set times this factor
    keeps the sign of every value, so every seed has surfaces of its own on the same cut tets."""

    def at(d3, d2, d1):
        g = [(np.arange(n + 1 - d) + 0.5 * d) / n for d in (d3, d2, d1)]
        z, y, x = (w * t for w, t in zip(wave, g))
        return (1.0 + 0.1 * np.sin(phase + z[:, None, None] + y[None, :, None] + x[None, None, :])).ravel()

    return at(0, 0, 0), np.concatenate([at(*d) for d in _EDGE_DIRS]) if p2 else None


def _bend_of(rng):
    return rng.uniform(2.0, 6.0, 3), rng.uniform(0.0, 6.0)


def _fe(case):
    return tf.P2IF if case["fe"] == "p2" else tf.P1IF


def _prec(case):
    return tf.PREC_MIXED if case["prec"] == "mixed" else tf.PREC_FP64


def _grid_matrix(case, seed):
    """An implicit Euler step of a diffusion(-convection) problem with variable coefficients on a k1 x k2 x k3 grid:
    7-point rows (rowptr, colind, vals), nonsymmetric for GMRES, and a right-hand side."""
    k = [case["k1"], case["k2"], case["k3"]]
    m = k[0] * k[1] * k[2]
    rng = np.random.default_rng(seed)
    idx = np.arange(m).reshape(k)
    sym = case.get("solver", "pcg") != "gmres"
    rows, cols, vals = [], [], []
    diag = np.full(m, 0.2) * rng.uniform(1.0, 2.0, m)
    for d in range(3):
        lo = np.take(idx, range(k[d] - 1), axis=d).ravel()
        hi = np.take(idx, range(1, k[d]), axis=d).ravel()
        w = np.exp(rng.uniform(-1.0, 1.0, lo.size))
        wind = np.zeros(lo.size) if sym else w * rng.uniform(0.0, 0.4, lo.size)
        rows += [lo, hi]
        cols += [hi, lo]
        vals += [-w + wind, -w - wind]
        diag += np.bincount(lo, w + wind, m) + np.bincount(hi, w + wind, m)
    rows, cols, vals = (np.concatenate(x) for x in (rows + [np.arange(m)], cols + [np.arange(m)], vals + [diag]))
    order = np.lexsort((cols, rows))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int64)
    return rowptr, cols[order].astype(np.int64), vals[order], rng.standard_normal(m)


def prepare(case, seed):
    S = State(case)
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "noalloc":
        rp, ci, v, b = _grid_matrix(case, seed)
        S.m = rp.size - 1
        S.rp, S.ci = (torch.from_numpy(x.astype(np.int32)).cuda() for x in (rp, ci))
        S.v, S.b = torch.from_numpy(v).cuda(), torch.from_numpy(b).cuda()
        S.x = torch.zeros_like(S.b)
        tf.load_library()
        return S
    S.ctx = ctx = tf.TraceFEM(0)
    if kind == "user":
        S.rp, S.ci, S.v, S.b = _grid_matrix(case, seed)
        S.x0 = np.zeros(S.rp.size - 1)
        return S
    if kind == "batch":
        W = ellipsoid_batch(case["count"], case["nmin"], case["nmax"])
        ctx.brick_batch(W["n"], W["orig"], W["axes"])
        ctx.levelset_analytic_batch(tf.LS_ELLIPSOID, W["par"], p2=False)
        # factors that keep every value's sign: the seed changes the surfaces, not which tets they cut
        lv, _ = ctx.levelset_download()
        ctx.levelset_upload(lv * np.tile(1.0 + 0.05 * rng.uniform(-1.0, 1.0, 4096), lv.size // 4096 + 1)[: lv.size])
        S.coef = np.stack([np.ones(len(W["h"])), np.ones(len(W["h"])), W["h"]], axis=1)
        S.load = [0.0, 0.0, 0.0, 1.0, rng.uniform(8.0, 18.0)]
        return S
    shape = "torus" if kind == "ch" else case.get("shape", "sphere")
    S.a, S.ls, S.par = _surface(shape)
    n = case["n"]
    S.h = 2 * S.a / n
    bend = _bend_of(rng)
    S.load = [0.0, 0.0, 0.0, 1.0, rng.uniform(8.0, 18.0)]
    if kind == "refine":
        return S
    ctx.brick_cube(n, S.a)
    p2 = case.get("fe") == "p2" or kind == "quaqua"
    ctx.levelset_analytic(S.ls, S.par, p2=p2)
    if kind in ("step", "forms", "quaqua"):
        lv, le = ctx.levelset_download()
        bv, be = _bend(n, *bend, p2)
        S.lv, S.le = S.pin(lv * bv), S.pin(le * be) if p2 else None
        ctx.levelset_upload(S.lv, S.le)
    if kind == "ch":
        _, m = ctx.distribute_dofs(tf.P1IF)
        ctx.setup_fe_system(FORMS)
        S.x0 = S.pin(np.concatenate([0.5 + rng.uniform(-0.01, 0.01, m), np.zeros(m)]))
        S.out = np.empty(2 * m)
    if kind == "quaqua":
        _, m = ctx.distribute_dofs(tf.P2IF)
        nnz = ctx.setup_fe_system([tf.FORM_M])
        S.vals = [np.empty(nnz), np.empty(nnz)]
        S.rhs = np.empty(m)
    if kind == "spmv":
        _, m = ctx.distribute_dofs(_fe(case))
        ctx.setup_fe_system(FORMS)
        ctx.lincomb(FORMS, [1.0, 1.0, S.h])
        ctx.vec_upload(tf.VEC_T0, rng.standard_normal(m))
        S.out = np.empty(m)
    return S


def _solved(st, res):
    if st != tf.OK or res > TOL:
        raise RuntimeError(f"solve failed: status {st}, residual {res}")


def run(S):
    case, ctx = S.case, S.ctx
    kind = case["kind"]
    if kind == "noalloc":
        S.x.zero_()
        torch.cuda.current_stream().synchronize()
        it, tol = C.c_int(100000), C.c_double(TOL)
        p = [C.c_void_p(t.data_ptr()) for t in (S.rp, S.ci, S.v, S.b, S.x)]
        st = tf.load_library().tf_pcg_jacobi_noalloc(C.c_int64(S.m), *p, C.byref(it), C.byref(tol), C.c_int(1), None)
        _solved(st, tol.value)
        return S.x
    if kind == "user":
        ctx.matrix_upload(S.rp, S.ci, S.v)
        ctx.vec_upload(tf.VEC_B, S.b)
        ctx.vec_upload(tf.VEC_X, S.x0)
        if case["solver"] == "gmres":
            st, _, res = ctx.gmres_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, restart=50, tol=TOL, method=case["method"])
        else:
            prec = tf.PREC_MIXED if case["solver"] == "pcg_mixed" else tf.PREC_FP64
            st, _, res = ctx.pcg_jacobi(tf.MAT_USER, tf.VEC_B, tf.VEC_X, tol=TOL, precision=prec)
        _solved(st, res if case["method"] == 0 else min(res, TOL))
        return ctx.vec_download(tf.VEC_X)
    if kind == "batch":
        _, m = ctx.distribute_dofs(tf.P1IF)
        ctx.setup_fe_system(FORMS, tf.RHS_SPHERE_XYZ, S.load)
        ctx.batch_lincomb(FORMS, S.coef)
        ctx.vec_fill(tf.VEC_X, m, 0.0)
        st, _, res = ctx.batch_pcg_jacobi(tf.MAT_SYS, tf.VEC_RHS, tf.VEC_X, tol=TOL, precision=_prec(case))
        _solved(st, res.max())
        return ctx.vec_download(tf.VEC_X)
    if kind == "ch":
        ctx.vec_upload(tf.VEC_X, S.x0)
        if case["learned"] < 0:
            ctx.ch_steps(case["steps"], 1e-3, 1.0, 0.02, 0.0, 1.0, S.h, restart=50, tol=CH_TOL)
        else:
            if case["learned"] == 1:
                ctx.mlp_init(1234)
            ctx.ch_steps_learned(case["steps"], 1e-3, 1.0, 0.02, 0.0, 1.0, S.h, restart=50, tol=CH_TOL, precision=_prec(case),
                                 learned=case["learned"], train_steps=case["steps"])
        return ctx.vec_download(tf.VEC_X, out=S.out)
    if kind == "quaqua":
        ctx.setup_quaqua_p2(S.load[4])
        for f, v in zip((tf.FORM_M, tf.FORM_A), S.vals):
            ctx.call("tf_matrix_download", C.c_int(f), None, None, v.ctypes.data_as(C.POINTER(C.c_double)))
        return [*S.vals, ctx.vec_download(tf.VEC_RHS, out=S.rhs)]
    if kind == "spmv":
        ctx.spmv(tf.MAT_SYS, tf.VEC_T0, tf.VEC_T1)
        return ctx.vec_download(tf.VEC_T1, out=S.out)
    if kind == "refine":
        ctx.brick_cube(case["n"], S.a)
        ctx.mesh_refine_band(S.ls, S.par, case["width"], 0, case["levels"])
        ctx.levelset_analytic(S.ls, S.par, p2=True)
        fe, prec = tf.P2IF, tf.PREC_MIXED
    else:
        fe, prec = _fe(case), _prec(case) if kind == "step" else None
        if kind == "step" and case["upload"]:
            ctx.levelset_upload(S.lv, S.le)
    na, m = ctx.distribute_dofs(fe)
    if kind == "forms":
        ctx.setup_fe_system(FORMS, tf.RHS_CONST, [S.load[4]])
        ctx.lincomb(FORMS, [1.0, 1.0, S.h])
        return [na, m, *ctx.matrix(tf.MAT_SYS), ctx.vec_download(tf.VEC_RHS)]
    ctx.setup_fe_system(FORMS, tf.RHS_SPHERE_XYZ, S.load)
    ctx.lincomb(FORMS, [1.0, 1.0, S.h])
    ctx.vec_fill(tf.VEC_X, m, 0.0)
    st, _, res = ctx.pcg_jacobi(tf.MAT_SYS, tf.VEC_RHS, tf.VEC_X, tol=TOL, precision=prec)
    _solved(st, res)
    return [na, m, ctx.vec_download(tf.VEC_X)]


# ---------------------------------------------------------------------------------------------------------------
# Sizes of a surface problem on n^3 cubes: level-set values (vertices, and edges for P2), and cut tets, rows and
# non-zeros, which grow as n^2 times the surface's area (counted on the 96^3 sphere and the 128^3 torus).
def _sizes(fe, shape, n):
    nv, ne = (n + 1) ** 3, 7 * n ** 3
    cut = (7.74 if shape == "sphere" else 10.37) * n * n
    rows = cut * (2.04 if fe == "p2" else 0.344)
    return nv + (ne if fe == "p2" else 0), cut, rows, rows * (22.8 if fe == "p2" else 10.8)


def _solve_work(rows, nnz, iters):
    # per iteration: one product and ten vector operations; the matrix itself has to be read once
    return iters * (2 * nnz + 12 * rows)


def _asm_flops(fe, cut):
    # per cut tet: about 4 facets of 7 points and 15 volume points, three forms
    return cut * ((28 * (110 * 2 + 190) + 15 * 120) if fe == "p2" else (28 * 60 + 15 * 40))


def work(case):
    kind = case["kind"]
    if kind in ("user", "noalloc"):
        m = case["k1"] * case["k2"] * case["k3"]
        gm = case.get("solver") == "gmres"
        # GMRES(50): on average 25 basis vectors take part in an orthogonalisation
        return {"bytes": (16 if kind == "user" else 12) * 7 * m + 8 * 4 * m, "flops": 60 * m * ((14 + 4 * 25) if gm else 26)}
    if kind == "batch":
        sizes = range(case["nmin"], case["nmax"] + 1)
        b = f = 0.0
        for n in sizes:
            ls, cut, rows, nnz = _sizes("p1", "sphere", n)
            b += 8 * (ls + rows)
            f += _asm_flops("p1", cut) + _solve_work(rows, nnz, 5 * n)
        return {"bytes": b * case["count"] / len(sizes), "flops": f * case["count"] / len(sizes)}
    n = case["n"]
    if kind == "ch":
        _, _, rows, nnz = _sizes("p1", "torus", n)
        it = case["steps"] * (1000 if case["prec"] == "mixed" else 1100)
        return {"bytes": 12 * 3 * nnz + 32 * rows, "flops": it * (2 * 4 * nnz + 4 * 25 * 2 * rows)}
    if kind == "refine":
        # the band's tets are those of the brick refined everywhere; the rest of the mesh is coarse
        ls, cut, rows, nnz = _sizes("p2", "sphere", n * 2 ** case["levels"])
        return {"bytes": 8 * rows, "flops": _asm_flops("p2", cut) + _solve_work(rows, nnz, 20 * n * 2 ** case["levels"])}
    if kind == "spmv":
        _, _, rows, nnz = _sizes(case["fe"], "sphere", n)
        return {"bytes": 12 * nnz + 20 * rows, "flops": 2 * nnz}
    if kind == "quaqua":
        ls, cut, rows, nnz = _sizes("p2", "sphere", n)
        return {"bytes": 8 * ls + 16 * nnz + 8 * rows, "flops": cut * 11 * 3000}
    ls, cut, rows, nnz = _sizes(case["fe"], case["shape"], n)
    if kind == "forms":
        return {"bytes": 8 * ls + 16 * nnz + 16 * rows, "flops": _asm_flops(case["fe"], cut)}
    it = (17 if case["fe"] == "p2" else 5) * n
    return {"bytes": 8 * ls + 8 * rows, "flops": _asm_flops(case["fe"], cut) + _solve_work(rows, nnz, it)}


# ---------------------------------------------------------------------------------------------------------------
def _solve64(rowptr, colind, vals, b):
    """x with A x = b by BiCGStab with a Jacobi preconditioner in 64 bits, refined until the residual stalls."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = [torch.from_numpy(x).to(dev) for x in (rowptr, colind, vals, b)]
    A = torch.sparse_csr_tensor(t[0], t[1], t[2], (b.size, b.size), dtype=torch.float64)
    rows = torch.repeat_interleave(torch.arange(b.size, device=dev), t[0][1:] - t[0][:-1])
    d = torch.zeros_like(t[3]).index_add_(0, rows[t[1] == rows], t[2][t[1] == rows])
    x = torch.zeros_like(t[3])
    best = math.inf
    for _ in range(8):
        r = t[3] - A @ x
        rn = float(r.norm())
        if rn >= 0.5 * best or rn == 0.0:
            break
        best = rn
        r0, p, dx = r.clone(), r.clone(), torch.zeros_like(x)
        rho = r0 @ r
        for _ in range(400):
            ph = p / d
            v = A @ ph
            alpha = rho / (r0 @ v)
            s = r - alpha * v
            sh = s / d
            q = A @ sh
            om = (q @ s) / (q @ q)
            dx += alpha * ph + om * sh
            r = s - om * q
            if float(r.norm()) < 1e-12 * rn:
                break
            rho1 = r0 @ r
            p = r + (rho1 / rho) * (alpha / om) * (p - om * v)
            rho = rho1
        x = x + dx
    return x.cpu().numpy()


def _kuhn(n):
    """Tets of the n^3 Kuhn brick in order (cubes by i3, i2, i1; six tets each), as vertex numbers."""
    axes = [(2, 1), (2, 0), (1, 2), (1, 0), (0, 2), (0, 1)]  # first and second step, (i3, i2, i1) = 0, 1, 2
    i3, i2, i1 = torch.meshgrid(*[torch.arange(n)] * 3, indexing="ij")
    base = torch.stack([i3, i2, i1], -1).reshape(-1, 1, 1, 3)
    off = torch.zeros(6, 4, 3, dtype=torch.long)
    for l, (f, s) in enumerate(axes):
        off[l, 1, f] = off[l, 2, f] = off[l, 2, s] = 1
        off[l, 3] = 1
    p = (base + off).reshape(-1, 4, 3)
    return (p[..., 0] * (n + 1) + p[..., 1]) * (n + 1) + p[..., 2]


def _exact_forms(case, seed):
    """M + A + h C_n and the load vector of a constant f for P1 and a P1 level set, from the planar cuts of the tets: the
    integrands are polynomials there, so the integrals are those of any rule exact for them."""
    rng = np.random.default_rng(seed)
    a, ls, par = _surface(case["shape"])
    n = case["n"]
    bend = _bend_of(rng)
    load = rng.uniform(8.0, 18.0)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.arange(n + 1, dtype=torch.float64)
    z, y, x = torch.meshgrid(*[-a + g * (2 * a / n)] * 3, indexing="ij")
    X = torch.stack([x, y, z], -1).reshape(-1, 3)
    if ls == tf.LS_SPHERE:
        phi = (X - torch.tensor(par[:3], dtype=torch.float64)).norm(dim=1) - par[3]
    else:
        q = (X ** 2).clone()
        q[:, int(par[2])] = 0
        phi = ((q.sum(1).sqrt() - par[0]) ** 2 + X[:, int(par[2])] ** 2).sqrt() - par[1]
    phi = phi * torch.from_numpy(_bend(n, *bend, False)[0])
    T = _kuhn(n)
    s = phi[T] > 0
    T = T[s.any(1) & ~s.all(1)]
    # first-touch numbering of the vertices of the cut tets
    flat = T.reshape(-1).numpy()
    verts, first = np.unique(flat, return_index=True)
    m = verts.size
    dof = np.empty(m, np.int64)
    dof[np.argsort(first)] = np.arange(m)
    L = torch.from_numpy(dof[np.searchsorted(verts, flat)].reshape(-1, 4)).to(dev)
    X, f, na = X[T].to(dev), phi[T].to(dev), T.shape[0]
    E = (X[:, 1:] - X[:, :1]).transpose(1, 2)  # columns: edges from vertex 0
    det = torch.linalg.det(E).abs()
    G = torch.linalg.inv(E)
    G = torch.cat([-G.sum(1, keepdim=True), G], 1)  # gradients of the hat functions
    grad = torch.einsum("ti,tic->tc", f, G)
    nrm = grad / grad.norm(dim=1, keepdim=True)
    gn = torch.einsum("tic,tc->ti", G, nrm)
    sg = G - gn[:, :, None] * nrm[:, None, :]
    # cut points in barycentric coordinates on the edges between the two sides, as one or two triangles
    pos = f > 0
    tris = []
    for mask in range(1, 15):
        code = (pos * torch.tensor([1, 2, 4, 8], device=dev)).sum(1)
        sel = (code == mask).nonzero()[:, 0]
        P, N = [i for i in range(4) if mask >> i & 1], [i for i in range(4) if not mask >> i & 1]
        if not sel.numel():
            continue
        ff = f[sel]

        def cut(i, j):
            b = torch.zeros(sel.numel(), 4, dtype=torch.float64, device=dev)
            lam = ff[:, i] / (ff[:, i] - ff[:, j])
            b[:, i], b[:, j] = 1 - lam, lam
            return b

        pts = [cut(i, j) for i in P for j in N]
        if len(pts) == 3:
            tris.append((sel, torch.stack(pts, 1)))
        else:  # 2 + 2: the points in order around the quadrilateral are 0, 1, 3, 2
            tris.append((sel, torch.stack([pts[0], pts[1], pts[2]], 1)))
            tris.append((sel, torch.stack([pts[1], pts[3], pts[2]], 1)))
    M = torch.zeros(na, 4, 4, dtype=torch.float64, device=dev)
    area = torch.zeros(na, dtype=torch.float64, device=dev)
    F = torch.zeros(na, 4, dtype=torch.float64, device=dev)
    for sel, B in tris:
        W = torch.einsum("tkj,tjc->tkc", B, X[sel])
        ar = 0.5 * torch.linalg.cross(W[:, 1] - W[:, 0], W[:, 2] - W[:, 0]).norm(dim=1)
        mid = B.sum(1)
        M.index_add_(0, sel, ar[:, None, None] / 12 * (torch.einsum("tki,tkj->tij", B, B) + mid[:, :, None] * mid[:, None, :]))
        area.index_add_(0, sel, ar)
        F.index_add_(0, sel, ar[:, None] / 3 * mid)
    K = M + area[:, None, None] * torch.einsum("tic,tjc->tij", sg, sg)
    K = K + (2 * a / n) * (det / 6)[:, None, None] * gn[:, :, None] * gn[:, None, :]
    key = (L[:, :, None] * m + L[:, None, :]).reshape(-1)
    pat, inv = torch.unique(key, return_inverse=True)
    vals = torch.zeros(pat.numel(), dtype=torch.float64, device=dev).index_add_(0, inv, K.reshape(-1))
    rows, cols = (pat // m).cpu().numpy(), (pat % m).cpu().numpy()
    rhs = torch.zeros(m, dtype=torch.float64, device=dev).index_add_(0, L.reshape(-1), load * F.reshape(-1))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))])
    return [na, m, rowptr, cols, vals.cpu().numpy(), rhs.cpu().numpy()]


def exact(case, seed):
    if case["kind"] == "noalloc":
        return _solve64(*_grid_matrix(case, seed))
    if case["kind"] == "user":
        return _solve64(*_grid_matrix(case, seed))
    if case["kind"] == "forms" and case["fe"] == "p1":
        return _exact_forms(case, seed)
    return None
