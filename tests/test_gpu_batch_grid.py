"""Batched CG on square 5-point grids (one cluster a system, vectors on chip)
against the general batched kernel (explicit cluster and CTA sizes)."""
import numpy as np
import pytest

import flecsolve_gb300 as fs
from flecsolve_gb300 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = fs.Context()
    yield c
    c.close()


def _batch(sides):
    A, off = P.block_diagonal([P.diffusion(2, s, seed=40 + k) for k, s in enumerate(sides)])
    return A, off, P.uniform(6, A.nrows)


# sides at the edges: one row; the rows a CTA takes in one pass (22^2 < 512 <
# 23^2); one and several CTAs; a last slice that is short; the full slices of a
# 16-CTA cluster (424^2 = 16 x 11,236 rows)
@pytest.mark.parametrize("sides,rtol", [((1, 2, 3, 5, 22, 23), 1e-10), ((32, 33, 45, 46, 64), 1e-10),
                                        ((106, 107, 131), 1e-10), ((424,), 1e-5)])
@pytest.mark.parametrize("zero_guess,head", [(True, None), (False, None), (True, 0.0)])
def test_grid_batch_matches_general(ctx, sides, rtol, zero_guess, head):
    A, off, b = _batch(sides)
    x0 = np.zeros(A.nrows) if zero_guess else P.uniform(8, A.nrows)
    S = A.to_scipy()
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    got = []
    for kw in (dict(), dict(cluster=1, threads=256)):
        vx = fs.Vector(ctx, x0)
        infos = fs.batch_cg(dA, off, vb, vx, maxiter=4000, rtol=rtol, use_zero_guess=zero_guess,
                            fp64_head=head, **kw)
        got.append((infos, vx.numpy()))
    assert fs.batch_format(dA, off) == "grid"
    for k in range(len(sides)):
        i, ref = got[0][0][k], got[1][0][k]
        assert i.status == ref.status == "converged_rtol", (k, i, ref)
        # the suite's bar on FP32 recurrences with FP64 replacement
        assert abs(i.iters - ref.iters) <= 3, (k, i.iters, ref.iters)
        lo, hi = off[k], off[k + 1]
        rr = np.linalg.norm(b[lo:hi] - S[lo:hi] @ got[0][1]) / np.linalg.norm(b[lo:hi])
        assert rr <= rtol * (1 + 1e-3), (k, rr)
        assert abs(i.rhs_norm - ref.rhs_norm) <= 1e-6 * ref.rhs_norm
        assert abs(i.res_norm_initial - ref.res_norm_initial) <= 1e-6 * ref.res_norm_initial


def test_grid_batch_special_systems(ctx):
    """A zero right-hand side stops at once; a system that is not finite ends
    without touching the others; a limit of iterations is kept."""
    A, off, b = _batch((40, 41, 42, 60))
    b[off[0]:off[1]] = 0.0
    b[off[1] + 7] = np.nan
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    for maxiter in (4000, 30, 0):
        got = []
        for kw in (dict(), dict(cluster=1, threads=256)):
            vx = fs.Vector(ctx, A.nrows)
            got.append((fs.batch_cg(dA, off, vb, vx, maxiter=maxiter, rtol=1e-9, **kw), vx.numpy()))
        (i, x), (ref, xr) = got
        assert [s.status for s in i] == [s.status for s in ref]
        assert i[0].iters == 0 and not x[off[0]:off[1]].any()
        assert all(abs(p.iters - q.iters) <= 3 for p, q in zip(i, ref))
        assert np.isfinite(x[off[2]:]).all()
        assert np.isfinite(x[off[1]:off[2]]).all() == np.isfinite(xr[off[1]:off[2]]).all()


def test_grid_batch_with_clusters_that_wait_for_room(ctx):
    """Far more 15-CTA clusters than the GPU holds at once, so that clusters
    start while others end and their CTAs start apart: every system meets its
    tolerance, and repeated calls return the same bits."""
    A, off, b = _batch([400] * 40)
    S = A.to_scipy()
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    xs = []
    for _ in range(3):
        vx = fs.Vector(ctx, A.nrows)
        infos = fs.batch_cg(dA, off, vb, vx, maxiter=4000, rtol=1e-5)
        assert all(i.status == "converged_rtol" for i in infos)
        xs.append(vx.numpy())
    r = b - S @ xs[0]
    for lo, hi in zip(off[:-1], off[1:]):
        assert np.linalg.norm(r[lo:hi]) <= 1e-5 * (1 + 1e-3) * np.linalg.norm(b[lo:hi])
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])


def test_batch_on_chip_says_which_kernel_ran(ctx):
    """Squares with sizes left to the library: on chip, one launch for each
    cluster size; explicit sizes and systems that are no squares: the general
    kernel."""
    A, off, b = _batch((20, 33, 131))
    dA, vb, vx = fs.CSR(ctx, A), fs.Vector(ctx, b), fs.Vector(ctx, A.nrows)
    run = lambda **kw: fs.batch_cg(dA, off, vb, vx, maxiter=50, rtol=1e-3, **kw)
    for kw, ran in ((dict(), True), (dict(cluster=2, threads=256), False), (dict(), True), (dict(cluster=1), False),
                    (dict(threads=512), False), (dict(cluster=2, threads=256, cluster_systems=1), False)):
        run(**kw)
        assert (fs.batch_on_chip(dA, off) > 0) == ran
        if ran:
            assert fs.batch_on_chip(dA, off) <= 3
            assert fs.batch_schedule(dA, off)[0] in (1, 2, 4, 8)
    M, moff = P.block_diagonal([P.diffusion(3, 9, seed=1), P.diffusion(2, 30, seed=2)])
    dM = fs.CSR(ctx, M)
    fs.batch_cg(dM, moff, fs.Vector(ctx, P.uniform(3, M.nrows)), fs.Vector(ctx, M.nrows), maxiter=50, rtol=1e-3)
    assert fs.batch_on_chip(dM, moff) == 0
