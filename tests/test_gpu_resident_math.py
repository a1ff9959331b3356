"""The resident kernels' scalar arithmetic against exact results: the quotients
that replace FP64 divisions, the threshold of the stopping tests, and the sums
in fixed point, over exponents at every cut-over, hard-to-round quotients,
subnormals, cancellation and values that are not finite.  The bounds asserted
are those that the comments in csrc/resident.cuh state."""
import ctypes as C
import math
from fractions import Fraction as F

import numpy as np
import pytest

from flecsolve_gb300 import build

pytestmark = pytest.mark.gpu

DIVIDE, QUOTIENT, QUOTIENT32, THRESHOLD, WIDEN = range(5)


@pytest.fixture(scope="module")
def rm():
    return C.CDLL(str(build.build_math_test()))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _binary(rm, op, a, b=None):
    a = np.ascontiguousarray(a, np.float64)
    b = np.ones_like(a) if b is None else np.ascontiguousarray(b, np.float64)
    out = np.empty_like(a)
    assert rm.rm_binary(op, a.size, _p(a), _p(b), _p(out)) == 0
    return out


def _same(x, y):
    return (x == y) | (np.isnan(x) & np.isnan(y))


def _hard(rng, count):
    """a, b of 53 bits with (2 q + 1) b = a 2^k +- 1: a / b lies within 2^-105
    of the middle of two doubles."""
    out = []
    while len(out) < count:
        b = int(rng.integers(2 ** 52, 2 ** 53)) | 1
        if len(out) % 3 == 0:
            b = 2 ** 53 - 1 - 2 * int(rng.integers(0, 2000))
        for k in (53, 54):
            for s in (1, -1):
                q = pow(b, -1, 2 ** k) * s % 2 ** k
                a = (q * b - s) >> k
                if 2 ** 53 <= q < 2 ** 54 and 2 ** 52 <= a < 2 ** 53:
                    out.append((float(a), float(b)))
    return np.array(out[:count]).T


# biased exponents at the cut-overs of the quotients, and between
EDGES = [0, 1, 2, 122, 123, 124, 522, 523, 524, 903, 1022, 1023, 1024, 1143, 1144, 1522, 1523, 1922, 1923,
         2045, 2046, 2047]


def _operands():
    rng = np.random.default_rng(7)
    h = _hard(rng, 20000)
    n = 200000
    m = rng.integers(0, 2 ** 52, size=(2, n), dtype=np.uint64)
    m[0, : n // 8] = 0                       # powers of two
    m[1, n // 16: n // 5] = 2 ** 52 - 1      # all ones
    e = rng.choice(EDGES, size=(2, n)).astype(np.uint64)
    e[:, n // 2:] = rng.integers(900, 1150, size=(2, n - n // 2))
    s = rng.integers(0, 2, size=(2, n), dtype=np.uint64)
    r = (m | e << np.uint64(52) | s << np.uint64(63)).view(np.float64)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1.7976931348623157e308])
    g = np.array(np.meshgrid(special, np.concatenate([special, [1.0, -3.0]]))).reshape(2, -1)
    scale = 2.0 ** rng.integers(-400, 400, size=h.shape)
    return np.concatenate([h, -h, h * scale, r, g, g[::-1]], axis=1)


def test_quotients(rm):
    a, b = _operands()
    with np.errstate(all="ignore"):
        want = a / b
    # correctly rounded
    assert _same(_binary(rm, QUOTIENT, a, b), want).all()
    # half a unit and 2^-36 of one
    got = _binary(rm, DIVIDE, a, b)
    off = np.flatnonzero(~_same(got, want))
    for i in off:
        exact = F(a[i]) / F(b[i])
        unit = F(float(np.spacing(min(abs(got[i]), abs(want[i])))))
        assert abs(F(got[i]) - exact) <= unit * (F(1, 2) + F(1, 2 ** 36)), (a[i], b[i])
    assert np.array_equal(np.signbit(got[~np.isnan(got)]), np.signbit(want[~np.isnan(want)]))


def test_quotient32(rm):
    a, b = _operands()
    ea, eb = ((x.view(np.uint64) >> np.uint64(52) & np.uint64(0x7ff)).astype(int) for x in (a, b))
    short = (ea > 0) & (ea < 2047) & (eb > 0) & (eb < 2047) & (abs(ea - eb) <= 120)
    got = _binary(rm, QUOTIENT32, a, b)
    with np.errstate(all="ignore"):
        q = a / b
        f = q.astype(np.float32)
        assert _same(got[~short], f[~short].astype(np.float64)).all()
        unit = np.spacing(np.abs(f[short])).astype(np.float64)
    assert short.sum() > 100000
    assert (np.abs(got[short] - q[short]) <= 0.5 * unit + (2.0 ** -40 + 2.0 ** -52) * np.abs(q[short])).all()


def test_threshold(rm):
    """The largest s with sqrt(s) < tol: a test of s against it is the test of
    the norm."""
    rng = np.random.default_rng(3)
    tol = np.concatenate([np.exp(rng.uniform(-360, 354, 100000)), 2.0 ** np.arange(-540, 512.0),
                          [5e-324, 1e-170, 1.5e-162, 1e-161, 1.3407807929942596e154, 1e200]])
    t = _binary(rm, THRESHOLD, tol)
    top = 1.7976931348623157e308
    with np.errstate(over="ignore"):
        assert (np.sqrt(t) < tol).all()
        assert ((t == top) | ~(np.sqrt(np.nextafter(t, np.inf)) < tol)).all()
    assert (_binary(rm, THRESHOLD, [0.0, -0.0, -1.0, np.nan, -np.inf]) < 0).all()
    assert _binary(rm, THRESHOLD, [np.inf])[0] == top


def test_widen(rm):
    bits = np.random.default_rng(4).integers(0, 2 ** 32, size=400000, dtype=np.uint64).astype(np.uint32)
    bits[:512] = (np.arange(512) << 23).astype(np.uint32)
    f = bits.view(np.float32)
    f = f[~np.isnan(f)].astype(np.float64)
    assert np.array_equal(_binary(rm, WIDEN, f).view(np.uint64), f.view(np.uint64))


def test_fix_double(rm):
    """(hi 2^16 + lo 2^-30) 2^(E - 1075) rounded to nearest, ties to even; to a
    unit where the result is subnormal."""
    rng = np.random.default_rng(5)
    n = 60000
    hi = rng.integers(-2 ** 55, 2 ** 55, size=n) >> rng.integers(0, 56, size=n)
    lo = rng.integers(0, 2 ** 46, size=n) >> rng.integers(0, 47, size=n)
    lo[:2000] = 0
    # ties, and their neighbours
    k = rng.integers(0, 8, size=8000)
    hi[2000:10000] = (rng.integers(2 ** 53, 2 ** 54, size=8000) | 1) << k % 2
    lo[2000:10000] = np.where(k < 4, 0, np.where(k < 6, 1, 2 ** 46 - 1))
    hi[10000:12000] = 0
    E = rng.integers(1, 2047, size=n).astype(np.int32)
    E[::7] = rng.choice([1, 2, 20, 60, 1075, 2000, 2040, 2046], size=E[::7].size)
    out = np.empty(n)
    hi, lo = hi.astype(np.int64), lo.astype(np.int64)
    assert rm.rm_fix_double(n, _p(hi), _p(lo), _p(E), _p(out)) == 0
    for h, l, e, o in zip(hi.tolist(), lo.tolist(), E.tolist(), out.tolist()):
        v, x = (h << 46) + l, e - 1075 - 30
        try:
            want = math.ldexp(float(v), x)
        except OverflowError:
            want = math.copysign(math.inf, v)
        if abs(want) >= 2.0 ** -1021:
            assert o == want, (h, l, e)
        else:
            assert abs(F(o) - F(v) * F(2) ** x) <= F(2) ** -1074, (h, l, e)


def _unit(v):
    """2^(E - 1075) of the largest value of each row (the last bit of a double
    of its exponent)."""
    return np.maximum(np.spacing(np.abs(v).max(axis=-1)), 5e-324)


def _sets(rng, groups, n, f32=False):
    """Rows of n values: one scale, scales apart, cancelling, subnormal."""
    t = np.float32 if f32 else np.float64
    lim = 30 if f32 else 290
    one = rng.uniform(-1, 1, (groups, n))
    wide = rng.uniform(-1, 1, (groups, n)) * 10.0 ** rng.uniform(-lim, lim, (groups, n))
    near = rng.uniform(-1, 1, (groups, n)) * 2.0 ** rng.integers(-90, 1, (groups, n))
    half = rng.uniform(-1, 1, (groups, n // 2))
    cancel = np.concatenate([half, -half * (1 + 2.0 ** -40 * rng.uniform(-1, 1, half.shape))], axis=1)
    tiny = rng.integers(-50, 50, (groups, n)) * (1.4e-45 if f32 else 5e-324)
    pos = rng.uniform(0.5, 1, (groups, n)) * (2.0 ** 100 if f32 else 2.0 ** 900)
    return [np.ascontiguousarray(rng.permuted(x, axis=1).astype(t)) for x in (one, wide, near, cancel, tiny, pos)]


def _special(rng, groups, n, t):
    v = rng.uniform(-1, 1, (groups, n)).astype(t)
    for i in range(groups):
        bad = [[np.inf], [-np.inf], [np.inf, -np.inf], [np.nan], [np.nan, np.inf], [np.inf, np.inf]][i % 6]
        v[i, rng.choice(n, len(bad), replace=False)] = bad
    return np.ascontiguousarray(v)


def _fsum(v):
    return np.array([math.fsum(r) for r in v.astype(np.float64)])


def _error(got, v):
    """|got - the exact sum| of each row."""
    return np.abs(_fsum(np.concatenate([v.astype(np.float64), -got[:, None]], axis=1)))


@pytest.mark.parametrize("f32", [False, True])
def test_warp_sum(rm, f32):
    """The values lose bits below 2^-30 of the largest one's unit (FP32: 2^-31
    of the FP32 unit); the sum is rounded once."""
    rng = np.random.default_rng(6)
    fn, n = (rm.rm_warp_sum32, 256) if f32 else (rm.rm_warp_sum64, 128)
    g, out = 400, np.empty(400)
    for v in _sets(rng, g, n, f32):
        assert fn(g, _p(v), _p(out)) == 0
        exact = _fsum(v)
        lost = n * _unit(v).astype(np.float64) * 2.0 ** (-31 if f32 else -30)
        assert (_error(out, v) <= 0.5 * np.spacing(np.abs(exact) + lost) + lost + 5e-324).all()
    v = _special(rng, g, n, np.float32 if f32 else np.float64)
    assert fn(g, _p(v), _p(out)) == 0
    with np.errstate(invalid="ignore"):
        assert _same(out, v.astype(np.float64).sum(axis=1)).all()


@pytest.mark.parametrize("G", [1, 31, 152, 160])
@pytest.mark.parametrize("f32", [False, True])
def test_grid_sum(rm, f32, G):
    """512 values a CTA.  FP64: a warp's sum rounded to an eighth of the unit of
    its largest value, a CTA's to the unit, the total once; no worse than a tree
    of FP64 additions where that rounds.  FP32: each value loses at most 2^-29 of
    the FP32 unit of the largest (a double's unit), a CTA's sum is rounded to
    eight of these."""
    rng = np.random.default_rng(8)
    fn = rm.rm_grid_sum32 if f32 else rm.rm_grid_sum64
    groups, n = 12, 512 * G
    out, one = np.empty(groups), np.empty(groups)
    for kind, v in enumerate(_sets(rng, groups, n, f32)):
        assert fn(groups, G, _p(v), _p(out), _p(one)) == 0
        # the unit that the sums are kept in: a double's of the largest value
        u = _unit(v.astype(np.float64))
        for got, x, ctas in ((out, v, G), (one, v[:, :512], 1)):
            exact = _fsum(x)
            err = _error(got, x)
            lost = (512 + 4 if f32 else 1.5) * (1 + 1e-6) * ctas * u
            assert (err <= lost + 0.5 * np.spacing(np.abs(exact) + lost)).all(), kind
            if kind in (0, 5) and not f32:
                tree = np.zeros((groups, 1 << (x.shape[1] - 1).bit_length()))
                tree[:, : x.shape[1]] = x
                while tree.shape[1] > 1:
                    tree = tree[:, ::2] + tree[:, 1::2]
                floor = 0.5 * np.spacing(np.abs(exact)).max()
                assert err.max() <= max(_error(tree[:, 0], x).max(), floor)
    v = _special(rng, groups, n, np.float32 if f32 else np.float64)
    assert fn(groups, G, _p(v), _p(out), _p(one)) == 0
    with np.errstate(invalid="ignore"):
        assert _same(out, v.astype(np.float64).sum(axis=1)).all()
