"""The bit-exact kernels' branch-free quotients (pk_quotient.cuh) against
CUDA's correctly rounded division, bit for bit, wherever they say that the
operands are in their range, and that they say so for numerators in
[2^-768, 2^256), denominators in [2^-260, 2^252) and zero numerators of quoz and quoc.  Van Leer's
mean 2 a b / (a + b) (mean) alike, for a + b < 2^100 and a normal result.  Below these
ranges the sums that quoa and the comparisons that quob are for.

Operands: random ones; divisors with significands at either end; quotients
as close to the midpoint of two doubles as they get (n 2^54 - d m = +-1 for an
odd 54-bit m: m the inverse of d modulo 2^54); and values outside the range,
which must be refused or divided correctly."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "native", "quotient_harness.cu")
CSRC = os.path.join(HERE, "..", "piernik_b200", "csrc")
DEPS = [SRC, os.path.join(CSRC, "pk_quotient.cuh"), os.path.join(CSRC, "pk_device.cuh")]
LIB = os.path.join(HERE, "native", "libquotient_harness.so")

pytestmark = pytest.mark.gpu


def _lib():
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(p) for p in DEPS):
        subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false",
                               "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", LIB, SRC])
    return C.CDLL(LIB)


def _eval(n, d):
    n, d = np.ascontiguousarray(n, float), np.ascontiguousarray(d, float)
    out = np.empty((n.size, 9))
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert _lib().quotient_eval(p(n), p(d), n.size, p(out)) == 0
    return out


def _check(n, d, all_ok):
    o = _eval(n, d)
    want = o[:, 6].copy().view(np.uint64)
    for k, name in enumerate(("quo", "quoz", "quoc")):
        ok = o[:, 3 + k] != 0
        if all_ok:
            assert ok[(n != 0) | (k > 0)].all(), name
        bad = ok & (o[:, k].copy().view(np.uint64) != want) & ((n != 0) | (k > 0))
        assert not bad.any(), (name, n[bad][:3], d[bad][:3], o[bad][:3])


def _scaled(rng, x):
    return np.ldexp(x * rng.choice([-1.0, 1.0], x.size), rng.integers(-200, 200, x.size))


def test_random_and_edge_significands(gpu_lib):
    rng = np.random.default_rng(5)
    m = 1 << 20
    _check(_scaled(rng, 1 + rng.random(m)), _scaled(rng, 1 + rng.random(m)), True)
    ends = np.concatenate([1 + np.arange(64) * 2.0**-52, 2 - np.arange(1, 65) * 2.0**-52])
    _check(np.repeat(ends, ends.size), np.tile(ends, ends.size), True)
    _check(1 + rng.random(ends.size * 4096), np.tile(ends, 4096), True)
    zeros = np.tile([0.0, -0.0], 4096)
    _check(zeros, _scaled(rng, 1 + rng.random(zeros.size)), True)


def test_far_ends_of_the_range(gpu_lib):
    rng = np.random.default_rng(8)
    m = 1 << 18
    n = np.ldexp(1 + rng.random(m), rng.choice([-768, -767, -700, 254, 255], m))
    d = np.ldexp(1 + rng.random(m), rng.choice([-260, -259, 250, 251], m))
    _check(n, d, True)


def test_absorbed_quotients(gpu_lib):
    """big - x, big + x and x <= big with x of quoa and quob are those with n / d,
    wherever they say so; and they say so for every small numerator next to an
    ordinary big, zeros among them."""
    rng = np.random.default_rng(12)
    m = 1 << 19
    n = np.ldexp(1 + rng.random(m), rng.integers(-1080, 20, m)) * rng.choice([-1.0, 0.0, 1.0, 1.0], m)
    d = np.ldexp(1 + rng.random(m), rng.integers(0, 40, m))
    big = np.ldexp(1 + rng.random(m), rng.integers(-800, 200, m)) * rng.choice([-1.0, 1.0], m)
    near = rng.random(m) < 0.3              # quotients about as large as big
    big = np.where(near, n / d * (1 + rng.integers(-3, 4, m) * 2.0**-52), big)
    ends = rng.random(m) < 0.2              # powers of two: half the spacing below them
    big = np.where(ends & ~near, np.ldexp(1.0, rng.integers(-500, 200, m)), big)
    out = np.empty((m, 8))
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    n, d, big = (np.ascontiguousarray(x) for x in (n, d, big))
    assert _lib().absorbed_eval(p(n), p(d), p(big), m, p(out)) == 0
    ok = out[:, 2] != 0
    for k in (0, 1):
        assert np.array_equal(out[ok, k].copy().view(np.uint64), out[ok, 3 + k].copy().view(np.uint64)), k
    okb = out[:, 6] != 0
    assert np.array_equal(out[okb, 5], out[okb, 7])
    plain = (np.abs(big) > 2.0**-430) & (np.abs(big) < 2.0**200)
    assert ok[plain].all() and okb[plain].all() and ok.mean() > 0.5


def test_van_leer_mean(gpu_lib):
    rng = np.random.default_rng(9)
    m = 1 << 18
    a = np.ldexp(1 + rng.random(m), rng.integers(-440, 60, m))
    b = np.where(rng.random(m) < 0.5, a * (1 + 1e-3 * rng.random(m)), np.ldexp(1 + rng.random(m), rng.integers(-440, 60, m)))
    s = rng.choice([-1.0, 1.0], m)
    n, d = 2.0 * (a * b), s * (a + b)
    o = _eval(n, d)
    assert (o[:, 8] != 0).all()
    assert np.array_equal(o[:, 7].copy().view(np.uint64), o[:, 6].copy().view(np.uint64))
    zero = _eval(np.zeros(4), np.ones(4))
    assert (zero[:, 8] != 0).all() and (zero[:, 7].copy().view(np.uint64) == 0).all()
    # (2^-950 over 2^-470 was refused while products went down to 2^-900 only)
    far = _eval([2.0**-1060, 2.0**150, np.inf, np.inf, 2.0**100], [2.0**-30, 2.0**100, np.inf, np.nan, np.nan])
    assert (far[:, 8] == 0).all()
    # products down to the smallest subnormal ones, results down to the smallest normal ones
    a = np.ldexp(1 + rng.random(m), rng.integers(-537, -400, m))
    b = np.where(rng.random(m) < 0.5, a * (1 + rng.random(m)), np.ldexp(1 + rng.random(m), rng.integers(-537, -500, m)))
    n, d = 2.0 * (a * b), a + b
    o = _eval(n, d)
    some = n != 0
    assert (o[some, 8] != 0).all() and some.sum() > m // 2
    assert np.array_equal(o[some, 7].copy().view(np.uint64), o[some, 6].copy().view(np.uint64))


@pytest.mark.parametrize("on", [1, 0])
def test_van_leer_half_slopes(gpu_lib, on):
    """The slopes that the sweeps take (groups of five components, zero at pencil
    ends) against half of the reference's expression in IEEE operations
    (fluxlimiters.F90:122-133): random differences, every pair of the edges, and
    groups of ordinary components with one or two whose operands (beyond 2^100, or
    with a subnormal result) send the group to its IEEE redo.  The plain slope_interior is the adjoint's and the oracle
    tests' too."""
    tiny, sub = np.finfo(float).tiny, np.finfo(float).smallest_subnormal
    edge = [0.0, sub, 3 * sub, tiny, 1.5 * tiny, 1e-200, 1e-140, 1e-110, 0.75, 1.0, np.nextafter(1.0, 2.0), 3.0, 1e31, 1e120,
            1e200, 2.0**1022, 2.0**1023, np.inf, np.nan]
    edge = np.array(edge + [-x for x in edge])
    rng = np.random.default_rng(10)
    m = 40000
    dl = rng.standard_normal((m, 5)) * 10.0 ** rng.integers(-3, 3, (m, 5))
    dr = np.where(rng.random((m, 5)) < 0.5, dl * (1 + 0.1 * rng.standard_normal((m, 5))), rng.standard_normal((m, 5)))
    a, b = np.repeat(edge, edge.size), np.tile(edge, edge.size)
    rows = np.arange(a.size)
    for k in (0, 3, 4):                    # each pair of edges in a group of ordinary differences
        dl[k * 8000 + rows, k], dr[k * 8000 + rows, k] = a, b
    dl[16000 + rows, 1], dr[16000 + rows, 1] = b, b
    dl[16000 + rows, 2], dr[16000 + rows, 2] = a, b
    dl[10000:12000], dr[12000:14000] = 0.0, -0.0
    got, want = np.empty_like(dl), np.empty_like(dl)
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    dl, dr = np.ascontiguousarray(dl), np.ascontiguousarray(dr)
    assert _lib().vanleer_eval(on, p(dl), p(dr), m, p(got), p(want)) == 0
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))
    assert (want != 0).any() == bool(on)


def test_quotients_next_to_a_midpoint(gpu_lib):
    rng = np.random.default_rng(6)
    n, d = [], []
    for b in [int(x) | 1 for x in rng.integers(1 << 52, 1 << 53, 40000)] + [(1 << 53) - 1 - 2 * k for k in range(2000)]:
        inv = pow(b, -1, 1 << 54)
        for m, r in ((inv, 1), ((1 << 54) - inv, -1)):       # b m = r modulo 2^54
            a = (b * m - r) >> 54
            if a > 0 and m >> 53:
                n.append(float(a))
                d.append(float(b))
    assert len(n) > 10000
    n, d = np.array(n), np.array(d)
    _check(n, d, True)
    _check(np.ldexp(n, -60), -d, True)


def test_operands_outside_the_range(gpu_lib):
    edge = [0.0, 5e-324, 1e-310, 2.3e-308, 1e-200, 2.0**-257, 2.0**-256, 1.0, 2.0**255, 2.0**256, 1e200, 1.7e308, np.inf, np.nan]
    edge = np.array(edge + [-x for x in edge])
    n, d = np.repeat(edge, edge.size), np.tile(edge, edge.size)
    o = _eval(n, d)
    for k in range(3):
        ok = o[:, 3 + k] != 0
        assert not ok[~np.isfinite(n) | ~np.isfinite(d) | (d == 0)].any()
        same = o[:, k].copy().view(np.uint64) == o[:, 6].copy().view(np.uint64)
        assert same[ok].all()
