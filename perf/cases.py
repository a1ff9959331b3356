"""What is timed: the solves, gradients and operator applies that a program
built on this framework spends its time in, each through the package's public
calls (``flecsolve_gb300`` and ``flecsolve_gb300.adjoint``).

Twelve listed cases cover the range from a solve whose vectors fit in a few
SMs' shared memory (launch and synchronisation latency count) to the 16.8 M
row system that streams from HBM; grids whose side is a multiple of 4 and odd
ones (which take another storage); FP64 and mixed precision; forward, adjoint
and gradient; stencil and irregular rows.  ``draw`` spreads sizes and options
over the same ranges.

Tolerances: FP64 CG and GMRES run to the repository's benchmark tolerance or
tighter.  The methods whose iterates depend on rounding (mixed precision,
BiCGSTAB, block and batched solves) run to the tight tolerance of the adjoint
solves (1e-12, ``DiffusionSolve``'s default; 1e-11 for the block solve), so
that two correct implementations agree far below any digit a user reads.
"""
import math

import numpy as np
import torch

import flecsolve_gb300 as fs
from flecsolve_gb300 import adjoint as ad
from flecsolve_gb300 import problems as P


def listed():
    return [
        # 2-D Poisson, 16 k rows, FP64 Jacobi CG: the reference's own default
        # test problem size; a solve is a few hundred tiny iterations
        dict(name="cg-poisson2d-128", kind="solve", method="cg", problem="poisson2d", n=128,
             rtol=1e-8, maxiter=5000),
        # an ordinary 3-D FP64 CG on an odd side (no 16-byte grid lines: the
        # symmetric storage's path), 0.46 M rows
        dict(name="cg-diffusion3d-77", kind="solve", method="cg", problem="diffusion3d", n=77,
             rtol=1e-8, maxiter=5000),
        # FP64 BiCGSTAB on an ordinary convection-diffusion system, 0.26 M rows
        dict(name="bicgstab-convdiff3d-64", kind="solve", method="bicgstab", problem="convdiff3d",
             n=64, rtol=1e-12, maxiter=5000),
        # FP64 restarted GMRES(30) on the small Poisson system
        dict(name="gmres30-poisson2d-128", kind="solve", method="gmres", problem="poisson2d", n=128,
             rtol=1e-10, maxiter=5000),
        # the headline system: 16.8 M rows, mixed-precision PCG
        dict(name="mixed-cg-diffusion3d-256", kind="solve", method="mixed_cg", problem="diffusion3d",
             n=256, rtol=1e-12, maxiter=5000),
        # mixed BiCGSTAB on the 7.1 M row convection-diffusion system
        dict(name="mixed-bicgstab-convdiff3d-192", kind="solve", method="mixed_bicgstab",
             problem="convdiff3d", n=192, rtol=1e-12, maxiter=10000),
        # mixed restarted GMRES(30) on 0.88 M rows of the same operator
        dict(name="mixed-gmres30-convdiff3d-96", kind="solve", method="mixed_gmres",
             problem="convdiff3d", n=96, rtol=1e-12, maxiter=20000),
        # many uneven systems in one call: 512 2-D systems of side 32..256
        dict(name="batch-512-systems", kind="batch", nsys=512, lo=32, hi=256, rtol=1e-12,
             maxiter=5000),
        # 16 right-hand sides of one operator, mixed block CG, 2.1 M rows
        dict(name="block16-laplace3d-128", kind="block", problem="laplace3d", n=128, mixed=True,
             rtol=1e-11, maxiter=2000),
        # an inverse problem's step: forward solve, adjoint solve and the
        # gradients w.r.t. right-hand side and all face coefficients, 128^3
        dict(name="adjoint-diffusion3d-128", kind="adjoint", n=128, rtol=1e-12),
        # backward-Euler heat, 64^3 x 200 steps, differentiated through all
        # steps with a checkpoint every 20: some 600 short solves in a row
        dict(name="heat-gradient-64x200", kind="heat", n=64, steps=200, checkpoint=20),
        # one SpMV over irregular rows (power-law lengths, random columns)
        dict(name="spmv-powerlaw-1048576", kind="spmv", n=1048576, dtype="f64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cg2d", "cg3d", "bicgstab", "gmres", "mixed_cg", "mixed_bicgstab",
                       "mixed_gmres", "batch", "block", "adjoint", "heat", "spmv"])
    # the spread of the cell coefficients (log-normal) and the largest cell
    # Peclet number of the convection-diffusion operators
    sigma, pe = round(rng.uniform(0.5, 1.0), 3), round(rng.uniform(0.5, 5.0), 3)
    if kind == "cg2d":
        return dict(kind="solve", method="cg", problem=rng.choice(["poisson2d", "diffusion2d"]),
                    n=_log_int(rng, 32, 512), rtol=1e-8, maxiter=5000, sigma=sigma)
    if kind == "cg3d":
        return dict(kind="solve", method="cg", problem="diffusion3d", n=_log_int(rng, 12, 160),
                    rtol=1e-8, maxiter=5000, sigma=sigma)
    if kind == "bicgstab":
        return dict(kind="solve", method="bicgstab", problem="convdiff3d", n=_log_int(rng, 12, 128),
                    rtol=1e-12, maxiter=5000, pe=pe)
    if kind == "gmres":
        return dict(kind="solve", method="gmres", problem="poisson2d", n=_log_int(rng, 32, 160),
                    rtol=1e-10, maxiter=10000)
    if kind == "mixed_cg":
        return dict(kind="solve", method="mixed_cg", problem="diffusion3d", n=_log_int(rng, 48, 255),
                    rtol=1e-12, maxiter=5000, sigma=sigma)
    if kind == "mixed_bicgstab":
        return dict(kind="solve", method="mixed_bicgstab", problem="convdiff3d",
                    n=_log_int(rng, 32, 160), rtol=1e-12, maxiter=10000, pe=pe)
    if kind == "mixed_gmres":
        return dict(kind="solve", method="mixed_gmres", problem="convdiff3d", n=_log_int(rng, 32, 95),
                    rtol=1e-12, maxiter=20000, pe=pe)
    if kind == "batch":
        hi = rng.randrange(64, 257)
        return dict(kind="batch", nsys=_log_int(rng, 32, 500), lo=32, hi=hi, rtol=1e-12, maxiter=5000,
                    sigma=sigma)
    if kind == "block":
        return dict(kind="block", problem=rng.choice(["laplace3d", "diffusion3d"]),
                    n=_log_int(rng, 32, 127), mixed=True, rtol=1e-11, maxiter=2000, sigma=sigma)
    if kind == "adjoint":
        return dict(kind="adjoint", n=_log_int(rng, 24, 127), rtol=1e-12, sigma=sigma)
    if kind == "heat":
        steps = rng.randrange(20, 200)
        return dict(kind="heat", n=_log_int(rng, 16, 63), steps=steps, checkpoint=20,
                    sigma=sigma)
    return dict(kind="spmv", n=_log_int(rng, 1 << 16, 1 << 20), dtype=rng.choice(["f64", "f32"]))


# ------------------------------------------------------------- inputs ----

def _matrix(case, seed):
    """Host CSR of a solve, and its right-hand side's length."""
    n, problem = case["n"], case["problem"]
    if problem == "poisson2d":
        return P.poisson2d(n)
    if problem == "laplace3d":
        return P.laplace3d(n)
    if problem == "diffusion2d":
        return P.diffusion(2, n, seed=7 * seed + 2, sigma=case.get("sigma", 1.0))
    if problem == "diffusion3d":
        return P.diffusion(3, n, seed=7 * seed + 2, sigma=case.get("sigma", 1.0))
    return P.convdiff3d(n, seed=7 * seed + 4, pe_max=case.get("pe", 5.0))


def _batch(case, seed):
    sides = P.randint(5, case["nsys"], case["lo"], case["hi"])
    base, sigma = 1000 * (seed + 1), case.get("sigma", 1.0)
    A, off = P.block_diagonal([P.diffusion(2, int(s), seed=base + k, sigma=sigma)
                               for k, s in enumerate(sides)])
    return A, off, P.uniform(9 * seed + 6, A.nrows)


def _powerlaw(case, seed):
    """The power-law matrix of ``problems.powerlaw`` (row lengths, random
    columns, values U[-1, 1], a dominant diagonal), generated on the GPU."""
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(11 * seed + 9)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-300)
    lens = (16.0 * u.pow(-1.0 / 1.6)).floor().clamp_max(2048.0).clamp_max(float(n)).long()
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=rowptr[1:])
    nnz = int(rowptr[-1])
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    col = torch.randint(0, n, (nnz,), generator=g, device="cuda")
    col = torch.where(col == rows, (col + 1) % n, col)
    val = torch.rand(nnz, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    first = rowptr[:-1]
    col[first] = torch.arange(n, device="cuda")
    val[first] = 1.0 + lens.double()
    x = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    return rowptr, col.int(), val, x


def _faces(case, seed):
    return P.faces_lognormal(3, case["n"], seed=13 * seed + 7, sigma=case.get("sigma", 1.0))


def _adjoint_inputs(case, seed):
    """Face coefficients, right-hand side and target on the GPU."""
    rows = case["n"] ** 3
    arrays = (_faces(case, seed), P.uniform(13 * seed + 8, rows), P.uniform(13 * seed + 9, rows))
    return [torch.from_numpy(a).cuda() for a in arrays]


def _heat_inputs(case, seed):
    """Face coefficients, initial state and target (host arrays, as the call
    takes them)."""
    rows = case["n"] ** 3
    return (_faces(case, seed), P.uniform(13 * seed + 8, rows, 0.0, 1.0),
            P.uniform(13 * seed + 9, rows, 0.0, 1.0))


_HEAT_DT = 1e-3


def prepare(case, seed):
    """The operator, bound solver and vectors a program holds before its call."""
    ctx = fs.Context(0)
    kind = case["kind"]
    if kind == "solve":
        A = _matrix(case, seed)
        dA = fs.CSR(ctx, A)
        b = fs.Vector(ctx, P.uniform(5 * seed + 3, A.nrows))
        x = torch.zeros(A.nrows, dtype=torch.float64, device="cuda")
        method = getattr(fs, case["method"])
        kw = dict(max_krylov_dim=30, restart=True) if "gmres" in case["method"] else {}
        s = method.settings(maxiter=case["maxiter"], rtol=case["rtol"], use_zero_guess=True, **kw)
        solver = method.solver(s, method.make_work(b))(fs.op.ref(dA), fs.op.jacobi)
        torch.cuda.synchronize()
        return dict(case=case, ctx=ctx, A=dA, b=b, x=x, xv=fs.Vector.wrap(ctx, A.nrows, x.data_ptr()),
                    solver=solver)
    if kind in ("batch", "block"):
        if kind == "batch":
            A, off, rhs = _batch(case, seed)
        else:
            A, off = _matrix(case, seed), None
            rhs = P.uniform(5 * seed + 3, 16 * A.nrows)
        dA = fs.CSR(ctx, A)
        x = torch.zeros(rhs.size, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return dict(case=case, ctx=ctx, A=dA, off=off, b=fs.Vector(ctx, rhs), x=x,
                    xv=fs.Vector.wrap(ctx, rhs.size, x.data_ptr()))
    if kind == "adjoint":
        n = case["n"]
        system = ad.DiffusionSolve(ctx, 3, n, rtol=case["rtol"])
        faces, b, target = _adjoint_inputs(case, seed)
        torch.cuda.synchronize()
        return dict(case=case, system=system, solve=ad.LinearSolve(), faces=faces.requires_grad_(),
                    b=b.requires_grad_(), target=target)
    if kind == "heat":
        system = ad.DiffusionSolve(ctx, 3, case["n"], scale=_HEAT_DT, shift=1.0)
        faces, u0, target = _heat_inputs(case, seed)
        return dict(case=case, system=system, faces=faces, u0=u0, target=target)
    rowptr, col, val, x = _powerlaw(case, seed)
    n = case["n"]
    A = fs.CSR(ctx, P.CSR(n, n, rowptr.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()))
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    x = x.to(dt)
    y = torch.zeros(n, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    return dict(case=case, ctx=ctx, A=A, x=x, y=y, xv=fs.Vector.wrap(ctx, n, x.data_ptr(), case["dtype"]),
                yv=fs.Vector.wrap(ctx, n, y.data_ptr(), case["dtype"]))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        state["solver"](state["b"], state["xv"])
        return state["x"]
    if kind == "batch":
        fs.batch_cg(state["A"], state["off"], state["b"], state["xv"], case["maxiter"], case["rtol"])
        return state["x"]
    if kind == "block":
        fs.block_cg(state["A"], state["b"], state["xv"], 16, case["maxiter"], case["rtol"],
                    mixed=case["mixed"])
        return state["x"]
    if kind == "adjoint":
        faces, b = state["faces"], state["b"]
        faces.grad = b.grad = None
        x = state["solve"].apply(faces, b, state["system"])
        (x - state["target"]).square().sum().backward()
        return dict(x=x.detach(), dfaces=faces.grad, db=b.grad)
    if kind == "heat":
        L, dfaces, du0 = ad.heat_loss_and_grad(state["system"], state["faces"], state["u0"],
                                               state["target"], case["steps"], case["checkpoint"])
        return dict(loss=L, dfaces=dfaces, du0=du0)
    state["A"].apply(state["xv"], state["yv"])
    return state["y"]


# -------------------------------------------------------------- floors ---

# CG iterations per unit of grid side to a residual of 1e-8 (Jacobi
# preconditioner; the counts grow linearly with the side and the digits),
# rounded; used for the floors only, as the fits of the other methods below.
_ITERS = {"poisson2d": 3.0, "diffusion2d": 3.6, "diffusion3d": 3.5, "laplace3d": 3.5}


def _cache():
    return 129e6  # L2: a working set below it need not be re-read from memory


def work(case):
    """Bytes and operations of one pass.  A Krylov solve reads its matrix
    (as a stencil's symmetric or general diagonals) and reads or writes each
    recurrence vector once per use and iteration when they exceed the L2;
    otherwise each input is read and each output written once."""
    kind = case["kind"]
    if kind == "spmv":
        # mean row length of the power law, 8 or 4 bytes a value, 4 a column
        s = 8 if case["dtype"] == "f64" else 4
        n = case["n"]
        nnz = 40.6 * n
        return {"bytes": nnz * (s + 4) + 4 * n + 2 * n * s, "flops": 2 * nnz}
    if kind == "heat":
        n3 = case["n"] ** 3
        solves = 3 * case["steps"]
        # some 4 CG iterations a solve, about 28 operations a row each
        return {"bytes": 8.0 * (6 * n3 + 2 * 3 * n3), "flops": solves * 4 * 28.0 * n3}
    if kind == "batch":
        # 60 bytes per row and FP32 iteration (three coefficients, five vectors)
        mean = (case["lo"] + case["hi"]) / 2
        rows = case["nsys"] * (mean * mean + (case["hi"] - case["lo"]) ** 2 / 12)
        its = 3.5 * (case["lo"] + case["hi"])
        per = 60.0 if rows * 60 > _cache() else 0.0
        return {"bytes": rows * (4 * 8 + 2 * 8 + per * its), "flops": rows * its * 26}
    n = case["n"]
    if kind == "adjoint":
        its = 1.5 * _ITERS["diffusion3d"] * n
        rows = float(n ** 3)
        # FP64: SpMV 6 streams, update 7, direction 4 a row and iteration
        per = 17 * 8.0 if rows * 17 * 8 > _cache() else 0.0
        return {"bytes": rows * (8 * 12 + 2 * its * per), "flops": 2 * its * rows * 28}
    if kind == "block":
        rows = float(n ** 3)
        its = 1.4 * 2.3 * n
        # FP32 blocks of 16: SpMM 2 blocks + 4 coefficients, update 6, direction 3
        per = 11 * 64.0 + 16 if rows * 64 * 4 > _cache() else 0.0
        return {"bytes": rows * (16 * 16 + its * per), "flops": its * rows * (5 * 512 + 14 * 16)}
    dim = 2 if "2d" in case["problem"] else 3
    rows = float(n ** dim)
    method = case["method"]
    digits = -math.log10(case["rtol"]) / 8
    s = 4.0 if method.startswith("mixed") else 8.0
    coef = (1 + dim) if "convdiff" not in case["problem"] else 1 + 2 * dim
    if "cg" in method and "bicg" not in method:
        its, streams, ops = _ITERS[case["problem"]] * n * digits, coef + 2 + 10 + (0 if s == 4 else 1), 28
    elif "bicg" in method:
        its, streams, ops = 1.2 * n ** 1.45 * digits, 2 * (coef + 2) + 14, 60
    else:
        m = 30
        its = (0.42 if dim == 3 else 0.105) * n * n * digits
        streams, ops = coef + 2 + 2 * (m / 2 + 2), 14 + 4 * m
    keep = rows * streams * s
    per = streams * s if keep > _cache() else 0.0
    return {"bytes": rows * (8 * (coef + 2) + its * per), "flops": its * rows * ops}


# -------------------------------------------------- 64-bit answers -------

def _sparse(rowptr, col, val, n):
    with_dev = [torch.as_tensor(a).cuda() for a in (rowptr, col, val)]
    return torch.sparse_csr_tensor(with_dev[0].long(), with_dev[1].long(), with_dev[2].double(),
                                   size=(n, n))


def _cg64(mul, dinv, B, tol, maxiter):
    """Jacobi CG on every column of B at once (plain torch, FP64)."""
    X = torch.zeros_like(B)
    R = B.clone()
    Z = dinv * R
    Pm = Z.clone()
    rho = (R * Z).sum(0)
    stop = tol * B.norm(dim=0)
    for it in range(maxiter):
        W = mul(Pm)
        pap = (Pm * W).sum(0)
        alpha = torch.where(pap > 0, rho / pap, torch.zeros_like(rho))
        X += alpha * Pm
        R -= alpha * W
        Z = dinv * R
        new = (R * Z).sum(0)
        beta = torch.where(rho > 0, new / rho, torch.zeros_like(rho))
        Pm = Z + beta * Pm
        rho = new
        if it % 8 == 7 and bool((R.norm(dim=0) <= stop).all()):
            break
    return X


def _spd64(mul, diag, B, passes=3):
    """A^-1 B by CG with refinement on the FP64 residual."""
    dinv = (1.0 / diag).unsqueeze(1)
    X = _cg64(mul, dinv, B, 1e-10, 20000)
    for _ in range(passes - 1):
        X += _cg64(mul, dinv, B - mul(X), 1e-5, 20000)
    return X


def _bicg64(mul, dinv, b, tol, maxiter):
    x = torch.zeros_like(b)
    r = b.clone()
    rt = r.clone()
    p = torch.zeros_like(b)
    v = torch.zeros_like(b)
    rho = alpha = omega = torch.ones((), dtype=torch.float64, device=b.device)
    stop = tol * b.norm()
    for it in range(maxiter):
        new = torch.dot(rt, r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
        ph = dinv * p
        v = mul(ph)
        alpha = rho / torch.dot(rt, v)
        s = r - alpha * v
        sh = dinv * s
        t = mul(sh)
        omega = torch.dot(t, s) / torch.dot(t, t)
        x += alpha * ph + omega * sh
        r = s - omega * t
        if it % 8 == 7:
            rn = r.norm()
            if not bool(torch.isfinite(rn)) or bool(rn <= stop):
                break
    return x


def _gen64(mul, diag, b):
    """A^-1 b of a nonsymmetric operator: BiCGSTAB refined on the FP64
    residual until that residual stops falling."""
    dinv = 1.0 / diag
    x = torch.zeros_like(b)
    best = float(b.norm())
    for _ in range(12):
        d = _bicg64(mul, dinv, b - mul(x), 1e-6, 4000)
        if not bool(torch.isfinite(d).all()):
            break
        res = float((b - mul(x + d)).norm())
        if res >= best:
            break
        x, best = x + d, res
        if best <= 2e-15 * float(b.norm()):
            break
    return x


def _stencil64(faces, n):
    """(mul, diag) of K(c) on an n^3 grid from its face coefficients."""
    m = n * n * (n + 1)
    cx = faces[:m].view(n, n, n + 1)
    cy = faces[m:2 * m].view(n, n + 1, n)
    cz = faces[2 * m:].view(n + 1, n, n)
    diag = cx[..., 1:] + cx[..., :-1] + cy[:, 1:] + cy[:, :-1] + cz[1:] + cz[:-1]

    def mul(x):
        u = x.view(n, n, n)
        y = diag * u
        y[..., 1:] -= cx[..., 1:-1] * u[..., :-1]
        y[..., :-1] -= cx[..., 1:-1] * u[..., 1:]
        y[:, 1:] -= cy[:, 1:-1] * u[:, :-1]
        y[:, :-1] -= cy[:, 1:-1] * u[:, 1:]
        y[1:] -= cz[1:-1] * u[:-1]
        y[:-1] -= cz[1:-1] * u[1:]
        return y.reshape(x.shape)

    return mul, diag.reshape(-1)


def _face_grad64(lam, x, n):
    """-(lam_a - lam_b)(x_a - x_b) over the faces, 0 outside the grid."""
    pad = torch.nn.functional.pad
    a, b = lam.view(n, n, n), x.view(n, n, n)
    out = []
    for dim, p in ((2, (1, 1)), (1, (0, 0, 1, 1)), (0, (0, 0, 0, 0, 1, 1))):
        out.append((-torch.diff(pad(a, p), dim=dim) * torch.diff(pad(b, p), dim=dim)).reshape(-1))
    return torch.cat(out)


def exact(case, seed):
    """What ``run`` computes, in plain torch at 64 bits."""
    kind = case["kind"]
    if kind == "spmv":
        rowptr, col, val, x = _powerlaw(case, seed)
        rows = torch.repeat_interleave(torch.arange(case["n"], device="cuda"), rowptr.diff())
        y = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
        return y.index_add_(0, rows, val * x[col.long()])
    if kind == "adjoint":
        n = case["n"]
        faces, b, target = _adjoint_inputs(case, seed)
        mul, diag = _stencil64(faces, n)
        x = _spd64(lambda v: mul(v[:, 0])[:, None], diag, b[:, None])[:, 0]
        lam = _spd64(lambda v: mul(v[:, 0])[:, None], diag, (2 * (x - target))[:, None])[:, 0]
        return dict(x=x, dfaces=_face_grad64(lam, x, n), db=lam)
    if kind == "heat":
        n = case["n"]
        faces, u0, target = (torch.from_numpy(a).cuda() for a in _heat_inputs(case, seed))
        kmul, kdiag = _stencil64(faces, n)

        def step(v):
            return _spd64(lambda w: w + _HEAT_DT * kmul(w[:, 0])[:, None], 1 + _HEAT_DT * kdiag,
                          v[:, None], passes=2)[:, 0]

        states = [u0]
        for _ in range(case["steps"]):
            states.append(step(states[-1]))
        d = states[-1] - target
        lam, g = 2 * d, torch.zeros_like(faces)
        for u in reversed(states[1:]):
            lam = step(lam)
            g += _HEAT_DT * _face_grad64(lam, u, n)
        return dict(loss=float(d @ d), dfaces=g.cpu().numpy(), du0=lam.cpu().numpy())
    if kind == "batch":
        A, _, rhs = _batch(case, seed)
    else:
        A = _matrix(case, seed)
        rhs = P.uniform(5 * seed + 3, A.nrows * (16 if kind == "block" else 1))
    M = _sparse(A.rowptr, A.col, A.val, A.nrows)
    diag = torch.from_numpy(A.diagonal()).cuda()
    b = torch.from_numpy(rhs).cuda()
    if kind == "solve" and "convdiff" in case["problem"]:
        return _gen64(lambda v: torch.mv(M, v), diag, b)
    if kind == "block":
        return _spd64(lambda V: torch.sparse.mm(M, V), diag, b.view(-1, 16)).reshape(-1)
    return _spd64(lambda V: torch.mv(M, V[:, 0])[:, None], diag, b[:, None])[:, 0]
