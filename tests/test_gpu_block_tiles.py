"""Mixed block CG's warp tiles (32 rows) at sizes around a tile, a warp and the
grid, on grid stencils and on column ids, and the stops that leave a solution
step pending."""
import numpy as np
import pytest

import flecsolve_gb300 as fs
from flecsolve_gb300 import problems as P

pytestmark = pytest.mark.gpu


def _band(n, seed):
    """A symmetric diagonally dominant band matrix that is no grid stencil."""
    rng = np.random.default_rng(seed)
    D = np.zeros((n, n))
    for d in (1, 3, 7):
        v = -rng.uniform(0.5, 1.5, size=max(n - d, 0))
        D += np.diag(v, d) + np.diag(v, -d)
    D += np.diag(0.1 + np.abs(D).sum(1))
    rows, cols = np.nonzero(D)
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    return P.CSR(n, n, rp, cols.astype(np.int32), D[rows, cols])


def _solve(ctx, A, b, mixed=True, **kw):
    dA = fs.CSR(ctx, A)
    vb, vx = fs.Vector(ctx, b), fs.Vector(ctx, b.size)
    x0 = kw.pop("x0", None)
    if x0 is not None:
        vx.upload(x0)
    info = fs.block_cg(dA, vb, vx, 16, kw.pop("maxiter", 400), kw.pop("rtol", 1e-8),
                       use_zero_guess=x0 is None, mixed=mixed, **kw)
    return info, vx.numpy().reshape(-1, 16)


MATS = [("band", n) for n in (31, 32, 33, 250, 257, 1000)] + [("diffusion2d", n) for n in (6, 16, 37, 64)] + \
       [("diffusion3d", n) for n in (4, 9, 20, 33)]


@pytest.mark.parametrize("jacobi", [True, False])
@pytest.mark.parametrize("kind,n", MATS)
def test_mixed_block_cg_residuals(ctx, kind, n, jacobi):
    """The reported residual is the true FP64 one, and from 1000 rows on it
    meets the tolerance in every column.  (Sixteen columns exhaust the Krylov
    space of a few hundred rows; a column that converged keeps iterating with
    the others and may drift there.)"""
    A = _band(n, n) if kind == "band" else P.diffusion(2 if "2d" in kind else 3, n, seed=n)
    b = P.uniform(11, 16 * A.nrows)
    info, x = _solve(ctx, A, b, jacobi=jacobi, maxiter=600)
    M, B = A.to_scipy(), b.reshape(-1, 16)
    rel = np.linalg.norm(B - M @ x, axis=0) / np.linalg.norm(B, axis=0)
    for j, i in enumerate(info):
        if A.nrows >= 1000:
            assert i.status == "converged_rtol" and rel[j] <= 1.01e-8
        assert i.res_norm_final == pytest.approx(rel[j] * np.linalg.norm(B[:, j]), rel=1e-3, abs=1e-12)


@pytest.mark.parametrize("maxiter", [1, 2, 5, 17])
def test_mixed_block_cg_stopped_early_keeps_its_steps(ctx, maxiter):
    """At maxiter the pending step is in x: the iterate of the FP64 block CG to
    FP32 rounding, and the reported residual is that of x."""
    A = P.diffusion(3, 14, seed=5)
    b, x0 = P.uniform(11, 16 * A.nrows), P.uniform(12, 16 * A.nrows)
    for guess in (None, x0):
        one, x1 = _solve(ctx, A, b, maxiter=maxiter, rtol=1e-12, x0=guess)
        ref, x2 = _solve(ctx, A, b, mixed=False, maxiter=maxiter, rtol=1e-12, x0=guess)
        assert {i.status for i in one} == {i.status for i in ref} == {"diverged_iters"}
        assert one[0].restarts == ref[0].restarts == maxiter
        # 17 block iterations amplify the rounding of FP32 (6e-8) by the
        # condition of the Gram matrices; 1e-3 holds with three digits to spare
        assert np.linalg.norm(x1 - x2) <= 1e-3 * np.linalg.norm(x2)
        B = b.reshape(-1, 16)
        r = np.linalg.norm(B - A.to_scipy() @ x1, axis=0)
        assert np.allclose([i.res_norm_final for i in one], r, rtol=1e-4)


def test_mixed_block_cg_into_a_view(ctx):
    """X at an 8-byte aligned address: the same bits as in an own vector."""
    A = P.diffusion(3, 12, seed=4)
    b = P.uniform(11, 16 * A.nrows)
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    own, big = fs.Vector(ctx, b.size), fs.Vector(ctx, b.size + 1)
    view = fs.Vector.wrap(ctx, b.size, big.device_ptr + 8)
    for x in (own, view):
        fs.block_cg(dA, vb, x, 16, 300, 1e-9, mixed=True)
    assert np.array_equal(own.numpy(), view.numpy())
