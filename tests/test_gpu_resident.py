"""Solves that run in one cooperative launch against the kernel-per-phase
loops, which the other index formats still take, at the sizes where the slices
and the shared memory end."""
import numpy as np
import pytest

import flecsolve_gb300 as fs
from flecsolve_gb300 import problems as P
from flecsolve_gb300._lib import FsError

pytestmark = pytest.mark.gpu


def _grid(nx, ny, nz, dims, seed, asym=0.0):
    """CSR of a variable-coefficient grid stencil (offsets 1, nx, nx ny),
    diagonally dominant; asym > 0 makes the two triangles differ."""
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    idx = np.arange(n)
    i, j, k = idx % nx, idx // nx % ny, idx // (nx * ny)
    rows, cols, vals = [], [], []
    for d, (off, has) in enumerate(((1, i < nx - 1), (nx, j < ny - 1), (nx * ny, k < nz - 1))):
        if d >= dims:
            continue
        r = idx[has]
        up = -np.exp(rng.normal(size=r.size))
        lo = up * (1.0 + asym * rng.uniform(-1, 1, size=r.size))
        rows += [r, r + off]
        cols += [r + off, r]
        vals += [up, lo]
    rows, cols, vals = (np.concatenate(a) for a in (rows, cols, vals))
    diag = np.full(n, 0.05)
    np.add.at(diag, rows, np.abs(vals))
    rows, cols, vals = (np.concatenate(a) for a in ((rows, idx), (cols, idx), (vals, diag)))
    order = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    return P.CSR(n, n, rp, cols[order].astype(np.int32), vals[order])


def _solve(ctx, A, b, method, coding, x0=None, jacobi=True, **kw):
    dA = fs.CSR(ctx, A)
    assert dA.index_coding(coding) is not None
    m = getattr(fs, method)
    s = m.settings(use_zero_guess=x0 is None, **kw)
    vb = fs.Vector(ctx, b)
    vx = fs.Vector(ctx, x0 if x0 is not None else A.nrows)
    before = ctx.launches
    slv = m.solver(s, m.make_work(vb))(fs.op.ref(dA), fs.op.jacobi if jacobi else fs.op.I)
    info = slv(vb, vx)
    return info, vx.numpy(), slv.history(), ctx.launches - before


# slices of 32 rows to several arrays of global memory: one CTA and less, a
# CTA boundary inside a line, one and more rows a thread, more rows than five
# arrays (856 k), four and two arrays of shared memory hold
SHAPES = [((4, 3, 2), 3), ((4, 2, 2), 3), ((63, 1, 1), 1), ((64, 1, 1), 1), ((65, 1, 1), 1), ((12, 11, 1), 2),
          ((100, 97, 1), 2), ((152, 64, 1), 2), ((153, 64, 1), 2), ((37, 41, 29), 3),
          ((64, 64, 64), 3), ((96, 96, 95), 3), ((128, 128, 80), 3), ((130, 128, 127), 3)]


@pytest.mark.parametrize("shape,dims", SHAPES)
def test_resident_cg_matches_the_phase_kernels(ctx, shape, dims):
    """The same CG in another summation order: equal iterations and status,
    the solution within the bar of the FP64 CG (1e-10)."""
    A = _grid(*shape, dims, seed=sum(shape))
    b = P.uniform(3, A.nrows)
    kw = dict(maxiter=400, rtol=1e-9)
    one, x1, h1, l1 = _solve(ctx, A, b, "cg", "grid", **kw)
    ref, x2, h2, l2 = _solve(ctx, A, b, "cg", "patterns", **kw)
    assert (one.status, one.iters) == (ref.status, ref.iters) and one.success()
    assert l1 < l2
    assert np.linalg.norm(x1 - x2) <= 1e-10 * np.linalg.norm(x2)
    assert h1.size == h2.size and np.allclose(h1, h2, rtol=1e-6)
    for f in ("res_norm_initial", "sol_norm_final", "rhs_norm"):
        assert getattr(one, f) == pytest.approx(getattr(ref, f), rel=1e-6)


@pytest.mark.parametrize("jacobi", [True, False])
@pytest.mark.parametrize("shape,dims", [((48, 40, 1), 2), ((36, 20, 17), 3), ((128, 120, 64), 3)])
def test_resident_cg_warm_start_and_early_stops(ctx, shape, dims, jacobi):
    A = _grid(*shape, dims, seed=5)
    b = P.uniform(4, A.nrows)
    x0 = P.uniform(9, A.nrows)
    one, x1, h1, _ = _solve(ctx, A, b, "cg", "grid", x0=x0, jacobi=jacobi, maxiter=400, rtol=1e-9)
    ref, x2, h2, _ = _solve(ctx, A, b, "cg", "patterns", x0=x0, jacobi=jacobi, maxiter=400, rtol=1e-9)
    assert one.status == ref.status
    assert one.sol_norm_initial == pytest.approx(ref.sol_norm_initial, rel=1e-6)
    # the same recurrence: rounding has not grown over the first 20 steps
    assert np.allclose(h1[:20], h2[:20], rtol=1e-9)
    if one.success():
        assert np.linalg.norm(b - A.to_scipy() @ x1) <= 1.001e-9 * np.linalg.norm(b)
    if jacobi:
        # without a preconditioner these coefficients let the order of a sum
        # move the count (303 to 305 at 48 x 40); with one the bar is 2
        assert abs(one.iters - ref.iters) <= 2
        if one.iters == ref.iters:
            assert np.linalg.norm(x1 - x2) <= 1e-10 * np.linalg.norm(x2)
    # no iteration allowed, too few, a right-hand side of zeros, a converged guess
    for kw, rhs, guess in ((dict(maxiter=0, rtol=1e-9), b, None), (dict(maxiter=3, rtol=1e-9), b, x0),
                           (dict(maxiter=50, rtol=1e-9), 0 * b, None), (dict(maxiter=50, rtol=1e-6), b, x2)):
        one, x1, h1, _ = _solve(ctx, A, rhs, "cg", "grid", x0=guess, jacobi=jacobi, **kw)
        ref, y2, h2, _ = _solve(ctx, A, rhs, "cg", "patterns", x0=guess, jacobi=jacobi, **kw)
        assert (one.status, one.iters) == (ref.status, ref.iters)
        assert h1.size == h2.size
        assert np.allclose(x1, y2, rtol=1e-9, atol=1e-12)


def test_resident_cg_reports_non_finite(ctx):
    A = _grid(40, 36, 1, 2, seed=1)
    b = P.uniform(4, A.nrows)
    b[7] = np.inf
    for coding in ("grid", "patterns"):
        with pytest.raises(FsError) as e:
            _solve(ctx, A, b, "cg", coding, maxiter=50, rtol=1e-9)
        assert e.value.status == 5


@pytest.mark.parametrize("n", [9, 32, 65])
def test_transpose_solve_of_a_symmetric_matrix_is_the_forward_solve(ctx, n):
    A = P.diffusion(3, n, seed=3)
    dA = fs.CSR(ctx, A)
    vb, vx, vt = fs.Vector(ctx, P.uniform(8, A.nrows)), fs.Vector(ctx, A.nrows), fs.Vector(ctx, A.nrows)
    slv = fs.cg.solver(fs.cg.settings(maxiter=2000, rtol=1e-10))(fs.op.ref(dA), fs.op.jacobi)
    a = slv(vb, vx)
    t = slv.apply_transpose(vb, vt)
    assert (a.status, a.iters) == (t.status, t.iters)
    assert np.array_equal(vx.numpy(), vt.numpy())
    # values that stop being symmetric take the column view again
    v = A.val.copy()
    v[1] *= 1.0 + 1e-3
    dA.update_values(v)
    slv.apply_transpose(vb, vt)
    r = vb.numpy() - P.CSR(A.nrows, A.ncols, A.rowptr, A.col, v).to_scipy().T @ vt.numpy()
    assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(vb.numpy())


# ------------------------------------------------------------- GMRES -----

GM_SHAPES = [((5, 1, 1), 1, 0.0), ((64, 1, 1), 1, 0.0), ((12, 11, 1), 2, 0.3), ((100, 97, 1), 2, 0.0),
             ((152, 64, 1), 2, 0.3), ((36, 41, 29), 3, 0.3), ((48, 48, 47), 3, 0.0), ((64, 64, 61), 3, 0.3),
             ((96, 96, 95), 3, 0.3)]


@pytest.mark.parametrize("side", ["right", "left"])
@pytest.mark.parametrize("shape,dims,asym", GM_SHAPES)
@pytest.mark.parametrize("method", ["gmres", "mixed_gmres"])
def test_resident_gmres_matches_the_staged_passes(ctx, method, shape, dims, asym, side):
    """Delayed CGS2 in one launch against the same recurrence in kernels (row
    patterns).  FP64: counts within 2 and the estimates of the first 20 steps
    equal to 1e-9 (rounding only); FP32 basis: the suite's bar of mixed GMRES
    (1.2x + 30).  Either way the reported residual is the true one."""
    A = _grid(*shape, dims, seed=sum(shape), asym=asym)
    b = P.uniform(3, A.nrows)
    kw = dict(maxiter=600, rtol=1e-8, max_krylov_dim=30, restart=True, ortho="dcgs2", pre_side=side)
    one, x1, h1, l1 = _solve(ctx, A, b, method, "grid", **kw)
    ref, x2, h2, l2 = _solve(ctx, A, b, method, "patterns", **kw)
    assert one.status == ref.status
    if shape[0] % 4 == 0 and A.nrows <= 450000:  # the FP32 basis's limit
        assert l1 < l2
    if method == "gmres":
        assert abs(one.iters - ref.iters) <= 2
        assert np.allclose(h1[:20], h2[:20], rtol=1e-9, atol=1e-13 * h2[0])
    else:
        assert one.iters <= 1.2 * ref.iters + 30
    if one.success() and side == "right":
        M = A.to_scipy()
        for x in (x1, x2):
            assert np.linalg.norm(b - M @ x) <= 1.01e-8 * np.linalg.norm(b)
    assert one.res_norm_initial == pytest.approx(ref.res_norm_initial, rel=1e-5)
    assert one.sol_norm_final == pytest.approx(np.linalg.norm(x1), rel=1e-5)


@pytest.mark.parametrize("method", ["gmres", "mixed_gmres"])
def test_resident_gmres_stops(ctx, method):
    """Few iterations, a cycle longer than maxiter, no restart, a warm start,
    a right-hand side of zeros: the staged passes' answers."""
    A = _grid(48, 44, 1, 2, seed=2, asym=0.2)
    b, x0 = P.uniform(3, A.nrows), P.uniform(4, A.nrows)
    for kw, rhs, guess in ((dict(maxiter=0), b, None), (dict(maxiter=1), b, None), (dict(maxiter=7), b, x0),
                           (dict(maxiter=31), b, None), (dict(maxiter=60), b, x0), (dict(maxiter=40), 0 * b, None)):
        kw = dict(kw, rtol=1e-10, max_krylov_dim=30, restart=True, ortho="dcgs2")
        one, x1, h1, _ = _solve(ctx, A, rhs, method, "grid", x0=guess, **kw)
        ref, x2, h2, _ = _solve(ctx, A, rhs, method, "patterns", x0=guess, **kw)
        assert (one.status, one.iters, one.restarts) == (ref.status, ref.iters, ref.restarts)
        assert h1.size == h2.size
        tol = 1e-9 if method == "gmres" else 1e-3
        assert np.linalg.norm(x1 - x2) <= tol * max(np.linalg.norm(x2), 1e-30)
    kw = dict(maxiter=20, rtol=1e-2, max_krylov_dim=20, restart=False, ortho="dcgs2")
    one, x1, _, _ = _solve(ctx, A, b, method, "grid", **kw)
    ref, x2, _, _ = _solve(ctx, A, b, method, "patterns", **kw)
    assert (one.status, one.iters) == (ref.status, ref.iters)


# ---------------------------------------------------------- BiCGSTAB -----

@pytest.mark.parametrize("jacobi", [True, False])
@pytest.mark.parametrize("shape,dims,asym", GM_SHAPES)
def test_resident_bicgstab_matches_the_phase_kernels(ctx, shape, dims, asym, jacobi):
    """The same recurrence: norms equal to 1e-9 over the first 4 iterations
    (BiCGSTAB amplifies the rounding of its dots from there on), the stopping
    test met by the true residual, counts within a quarter of each other."""
    A = _grid(*shape, dims, seed=sum(shape), asym=asym)
    b, x0 = P.uniform(3, A.nrows), P.uniform(6, A.nrows)
    for guess in (None, x0):
        kw = dict(maxiter=600, rtol=1e-8, x0=guess, jacobi=jacobi)
        one, x1, h1, l1 = _solve(ctx, A, b, "bicgstab", "grid", **kw)
        ref, x2, h2, l2 = _solve(ctx, A, b, "bicgstab", "patterns", **kw)
        if shape[0] % 4 == 0:
            assert l1 < l2
        m = min(4, h1.size, h2.size)
        assert np.allclose(h1[:m], h2[:m], rtol=1e-9, atol=1e-12 * h2[0])
        assert one.res_norm_initial == pytest.approx(ref.res_norm_initial, rel=1e-6)
        if one.success() and ref.success():
            M = A.to_scipy()
            bn = np.linalg.norm(b)
            for x in (x1, x2):
                assert np.linalg.norm(b - M @ x) <= 2e-8 * bn
            assert abs(one.iters - ref.iters) <= 2 + 0.25 * ref.iters
        assert one.sol_norm_final == pytest.approx(np.linalg.norm(x1), rel=1e-5)


def test_resident_bicgstab_stops(ctx):
    """No iteration, few, zeros, the unscaled early exit at a loose rtol, a
    breakdown (r~'A P r = 0): the phase kernels' answers."""
    A = _grid(48, 44, 1, 2, seed=2, asym=0.2)
    b, x0 = P.uniform(3, A.nrows), P.uniform(4, A.nrows)
    for kw, rhs, guess in ((dict(maxiter=0, rtol=1e-9), b, None), (dict(maxiter=3, rtol=1e-9), b, x0),
                           (dict(maxiter=20, rtol=1e-9), 0 * b, None), (dict(maxiter=50, rtol=0.5), b, None),
                           (dict(maxiter=50, rtol=0.9), 1e-3 * b, None)):
        one, x1, h1, _ = _solve(ctx, A, rhs, "bicgstab", "grid", x0=guess, **kw)
        ref, x2, h2, _ = _solve(ctx, A, rhs, "bicgstab", "patterns", x0=guess, **kw)
        assert (one.status, one.iters) == (ref.status, ref.iters)
        assert h1.size == h2.size
        assert np.linalg.norm(x1 - x2) <= 1e-9 * max(np.linalg.norm(x2), 1e-30)


@pytest.mark.parametrize("shape,dims,asym", [((12, 11, 1), 2, 0.3), ((16, 32, 1), 2, 0.0), ((48, 44, 1), 2, 0.3),
                                             ((36, 20, 17), 3, 0.3)])
@pytest.mark.parametrize("method,u", [("gmres", 2.0 ** -53), ("mixed_gmres", 2.0 ** -24)])
def test_resident_gmres_estimate_is_the_true_residual(ctx, method, u, shape, dims, asym):
    """Every Hessenberg column and rotation: stopped after k steps, the
    estimate is the norm of b - A x_k.  A P V = V H + E with 8 + 2 (k + 1)
    roundings an entry in SpMV and update and |A D^-1| <= 2, so the two differ by
    at most 4 (k + 5) u (sqrt(k) |y| + estimate), |y| = |D x|; four times that
    for the norms formed from dots.  Solves repeat bit for bit."""
    A = _grid(*shape, dims, seed=sum(shape), asym=asym)
    b = P.uniform(3, A.nrows)
    M = A.to_scipy()
    D = M.diagonal()
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    assert dA.index_coding("grid") is not None
    ns = getattr(fs, method)
    first = None
    for k in list(range(1, 32)) + [31, 31]:
        s = ns.settings(use_zero_guess=True, maxiter=k, rtol=1e-30, max_krylov_dim=30, restart=True, ortho="dcgs2")
        vx = fs.Vector(ctx, A.nrows)
        slv = ns.solver(s, ns.make_work(vb))(fs.op.ref(dA), fs.op.jacobi)
        slv(vb, vx)
        h, x = slv.history(), vx.numpy()
        assert h.size == k
        if k < 31:
            true = np.linalg.norm(b - M @ x)
            bound = 16 * (k + 5) * u * (np.sqrt(k) * np.linalg.norm(D * x) + h[-1])
            assert abs(h[-1] - true) <= bound, (k, h[-1], true, bound)
        elif first is None:
            first = h, x
        else:
            assert np.array_equal(h, first[0]) and np.array_equal(x, first[1])


# ---------------------------------------------------- values not finite ---

GM = dict(max_krylov_dim=30, restart=True)


@pytest.mark.parametrize("coding", ["grid", "patterns"])
@pytest.mark.parametrize("method,kw", [("gmres", dict(GM, ortho=o, pre_side=p))
                                       for o in ("auto", "mgs", "cgs2", "dcgs2") for p in ("right", "left")] +
                         [("mixed_gmres", dict(GM, ortho=o)) for o in ("auto", "cgs2")] +
                         [("bicgstab", dict()), ("mixed_bicgstab", dict())])
def test_gmres_and_bicgstab_report_non_finite(ctx, method, kw, coding):
    """A NaN or an infinity in the matrix, the right-hand side or the guess
    ends every solver with the non-finite status (5), never as converged."""
    A = _grid(40, 36, 1, 2, seed=1, asym=0.2)
    b, x0 = P.uniform(4, A.nrows), P.uniform(9, A.nrows)
    at = int(np.flatnonzero(A.col == 700)[1])
    for bad in (np.nan, np.inf):
        v = A.val.copy()
        v[at] = bad
        B = P.CSR(A.nrows, A.ncols, A.rowptr, A.col, v)
        c, y0 = b.copy(), x0.copy()
        c[7] = y0[9] = bad
        for M, rhs, guess in ((B, b, None), (B, b, x0), (A, c, None), (A, c, x0), (A, b, y0)):
            with pytest.raises(FsError) as e:
                _solve(ctx, M, rhs, method, coding, x0=guess, maxiter=90, rtol=1e-9, **kw)
            assert e.value.status == 5


# ------------------------------------ an exact breakdown after a restart ---

def _breakdown(n):
    """GMRES(1) on this matrix leaves an exact eigenvector after its first
    cycle, every product and sum of both cycles being exact: |H(1, 0)| = 0 in
    the second.  A 1-D stencil that couples row 0 to row 1 alone."""
    A = _grid(n, 1, 1, 1, seed=1, asym=0.5)
    rows = np.repeat(np.arange(n), np.diff(A.rowptr))
    v = np.where(rows == A.col, 2.0, 0.0)
    v[0] = 1.0
    v[1] = -1.0
    return P.CSR(n, n, A.rowptr, A.col, v)


@pytest.mark.parametrize("n", [16, 256, 4096])
@pytest.mark.parametrize("route", ["grid", "patterns", "mgs", "cgs2", "shell"])
def test_gmres_exact_breakdown_in_the_second_cycle(ctx, n, route):
    """The estimate of a column without a rotation is 0, not the one that the
    cycle before left: converged after two iterations, on every route."""
    A = _breakdown(n)
    b = np.ones(n)
    dA, vb, vx = fs.CSR(ctx, A), fs.Vector(ctx, b), fs.Vector(ctx, n)
    dA.index_coding("grid" if route == "grid" else "patterns")
    op = fs.op.make_shell(ctx, lambda x, y: dA.apply(x, y), n) if route == "shell" else fs.op.ref(dA)
    ortho = dict(ortho=route) if route in ("mgs", "cgs2") else dict(ortho="dcgs2")
    s = fs.gmres.settings(maxiter=10, rtol=1e-12, use_zero_guess=True, max_krylov_dim=1, restart=True, **ortho)
    slv = fs.gmres.solver(s, fs.gmres.make_work(vb))(op, fs.op.I)
    info = slv(vb, vx)
    assert (info.status, info.iters, info.restarts) == ("converged_rtol", 2, 1)
    assert np.array_equal(A.to_scipy() @ vx.numpy(), b)


# ------------------------------- BiCGSTAB's breakdowns and its restart ---

# 4 x 4 tridiagonal blocks and right-hand sides on which the first iteration is
# exact (dyadic numbers): (a, b, what it meets)
BI_BLOCKS = {
    # skew: r~'A r = 0
    "alpha": ([[0, 1, 0, 0], [-1, 0, 0, 0], [0, 0, 0, 1], [0, 0, -1, 0]], [1, 1, 1, 1]),
    # t's = 0, t't = 3: omega = 0
    "omega": ([[-.5, 0, 0, 0], [0, 1.5, 0, 0], [0, 0, 1.5, 0], [0, 0, 0, 1.5]], [1, 1, 1, 1]),
    # r~'res = 0 after one iteration: restart from the true residual
    "restart": ([[-2, -1, 0, 0], [2, -1, 0, 0], [0, 1, 1, 1], [0, 0, -1, 0]], [1, -1, 1, -1]),
    "restart-2": ([[2, 0, 0, 0], [-3, -.5, 1, 0], [0, 3, 0, 0], [0, 0, 0, 1]], [-1, 2, 2, 2]),
}


def _blocks(kind, copies):
    a, b = BI_BLOCKS[kind]
    n = 4 * copies
    A = _grid(n, 1, 1, 1, seed=1, asym=0.5)
    rows = np.repeat(np.arange(n), np.diff(A.rowptr))
    same = rows // 4 == A.col // 4
    v = np.where(same, np.array(a)[rows % 4, A.col % 4], 0.0)
    return P.CSR(n, n, A.rowptr, A.col, v), np.tile(np.array(b, np.float64), copies)


@pytest.mark.parametrize("copies", [4, 64, 1024])
@pytest.mark.parametrize("kind", sorted(BI_BLOCKS))
def test_resident_bicgstab_breakdowns_and_restart(ctx, kind, copies):
    """r~'A P r = 0, omega = 0 and the restart at r~'res = 0, each met exactly:
    the error of the first, else the phase kernels' status, counts, restarts and solution, after every
    number of iterations up to 5, from a zero and a given guess, and the
    stopping test met by the true residual where a solve converges."""
    A, b = _blocks(kind, copies)
    M = A.to_scipy()
    x0 = np.ones(A.nrows)
    for guess, rhs in ((None, b), (x0, b + M @ x0)):
        for maxiter in (1, 2, 3, 4, 5, 200):
            kw = dict(maxiter=maxiter, rtol=1e-8, x0=guess, jacobi=False)
            if kind == "alpha":
                for coding in ("grid", "patterns"):
                    with pytest.raises(FsError, match="alpha = 0"):
                        _solve(ctx, A, rhs, "bicgstab", coding, **kw)
                continue
            one, x1, h1, l1 = _solve(ctx, A, rhs, "bicgstab", "grid", **kw)
            ref, x2, h2, l2 = _solve(ctx, A, rhs, "bicgstab", "patterns", **kw)
            assert l1 < l2
            assert one.status == ref.status
            if maxiter <= 5:
                assert (one.iters, one.restarts, h1.size) == (ref.iters, ref.restarts, h2.size)
                assert np.allclose(h1, h2, rtol=1e-9, atol=1e-12 * np.linalg.norm(b))
                assert np.allclose(x1, x2, rtol=1e-9, atol=1e-9)
            if kind == "omega":
                assert (one.status, one.iters, h1.size) == ("diverged_breakdown", 1, 1)
            elif maxiter > 1:
                assert one.restarts >= 1
            if one.success():
                assert np.linalg.norm(rhs - M @ x1) <= 2e-8 * np.linalg.norm(rhs)


# ------------------------------------------------- waits that run out ----

@pytest.mark.parametrize("method,kw", [("cg", {}), ("bicgstab", {}), ("gmres", GM), ("mixed_gmres", GM)])
@pytest.mark.parametrize("shape,dims,lost", [((12, 40, 1), 2, 0), ((128, 128, 1), 2, 77)])
def test_waits_that_run_out_end_the_solve_with_an_error(ctx, method, kw, shape, dims, lost):
    """A CTA that leaves at once sends no message: the others give up after
    their limit, an error and not a hang.  The next solve has the bits of a
    solver that never failed, whatever the failed one left behind."""
    A = _grid(*shape, dims, seed=3)
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, P.uniform(3, A.nrows))
    assert dA.index_coding("grid") is not None
    m = getattr(fs, method)
    s = m.settings(use_zero_guess=True, maxiter=60, rtol=1e-9, **kw)
    make = lambda: m.solver(s, m.make_work(vb))(fs.op.ref(dA), fs.op.jacobi)
    fresh, slv = make(), make()
    want, got = fs.Vector(ctx, A.nrows), fs.Vector(ctx, A.nrows)
    ref = fresh(vb, want)
    slv(vb, got)
    slv.lose_cta(lost)
    with pytest.raises(FsError, match="wait ran out"):
        slv(vb, got)
    slv.lose_cta(-1)
    for _ in range(2):
        info = slv(vb, got)
        assert (info.status, info.iters) == (ref.status, ref.iters)
        assert np.array_equal(got.numpy(), want.numpy())
        assert np.array_equal(slv.history(), fresh.history())


@pytest.mark.parametrize("shape", [(75, 77, 77), (75, 71, 73), (33, 35, 37)])
@pytest.mark.parametrize("method,u", [("gmres", 2.0 ** -53), ("mixed_gmres", 2.0 ** -24)])
def test_resident_gmres_estimate_on_odd_rows(ctx, method, u, shape):
    """As test_resident_gmres_estimate_is_the_true_residual, on row counts that
    are no multiple of 4 (the last group of four FP32 rows is short), most of
    whose columns are in global memory, and into the second cycle."""
    A = _grid(*shape, 3, seed=sum(shape))
    b = P.uniform(3, A.nrows)
    M = A.to_scipy()
    D = M.diagonal()
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    assert dA.index_coding("grid") is not None and A.nrows % 4
    ns = getattr(fs, method)
    for k in (1, 2, 13, 14, 15, 16, 29, 30, 37):
        s = ns.settings(use_zero_guess=True, maxiter=k, rtol=1e-30, max_krylov_dim=30, restart=True, ortho="dcgs2")
        vx = fs.Vector(ctx, A.nrows)
        before = ctx.launches
        slv = ns.solver(s, ns.make_work(vb))(fs.op.ref(dA), fs.op.jacobi)
        slv(vb, vx)
        assert ctx.launches - before < 8  # one launch, and the storage's
        h, x = slv.history(), vx.numpy()
        assert h.size == k
        true = np.linalg.norm(b - M @ x)
        bound = 16 * (min(k, 30) + 5) * u * (np.sqrt(min(k, 30)) * np.linalg.norm(D * x) + h[-1])
        assert abs(h[-1] - true) <= bound, (k, h[-1], true, bound)
