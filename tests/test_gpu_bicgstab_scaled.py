"""Mixed BiCGSTAB on grid stencils with asymmetric values, whose right Jacobi
preconditioning sits in a scaled copy of the values."""
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


def _line(n):
    rp = np.concatenate([[0], np.cumsum([2] + [3] * (n - 2) + [2])])
    col = np.concatenate([np.arange(max(r - 1, 0), min(r + 2, n)) for r in range(n)])
    val = np.where(col == np.repeat(np.arange(n), np.diff(rp)), 2.5, -1.0)
    return P.CSR(n, n, rp.astype(np.int32), col.astype(np.int32), val)


def _matrix(kind, n, seed):
    A = {1: _line, 2: P.poisson2d, 3: P.laplace3d}[kind](n)
    # rows scaled by different factors: the pattern of a grid, values not symmetric
    w = 1.0 + 9.0 * np.random.default_rng(seed).random(A.nrows)
    return P.CSR(A.nrows, A.ncols, A.rowptr, A.col, A.val * np.repeat(w, np.diff(A.rowptr)))


# 1-D, 2-D and 3-D grids (lines of one and of many 4-row segments), and a line
# length that the grid storage does not take
@pytest.mark.parametrize("kind,n", [(1, 16), (1, 64), (2, 8), (2, 36), (2, 37), (3, 4), (3, 12), (3, 40)])
def test_scaled_values(ctx, kind, n):
    A = _matrix(kind, n, 1)
    b = P.uniform(5, A.nrows)
    dA, vb = fs.CSR(ctx, A), fs.Vector(ctx, b)
    st = fs.mixed_bicgstab.settings(maxiter=2000, rtol=1e-10, use_zero_guess=True)
    slv = fs.mixed_bicgstab.solver(st, fs.mixed_bicgstab.make_work(vb))(fs.op.ref(dA), fs.op.jacobi)
    for seed in (1, 2):
        if seed == 2:
            # the same solver after a change of the values
            A = _matrix(kind, n, seed)
            dA.update_values(A.val)
        vx = fs.Vector(ctx, A.nrows)
        info = slv.apply(vb, vx)
        rr = np.linalg.norm(b - A.to_scipy() @ vx.numpy())
        assert info.status == "converged_rtol", info
        # the stopping test is on the FP64 residual
        assert rr <= 1e-10 * np.linalg.norm(b) * (1 + 1e-3)
        assert abs(info.res_norm_final - rr) <= 1e-3 * rr + 1e-13 * np.linalg.norm(b)
