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
