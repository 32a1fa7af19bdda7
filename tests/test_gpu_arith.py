"""The scalar arithmetic of the FP64 kernels (ec2d_dev.cuh, k_turb.cu) against IEEE
arithmetic and extended precision, operation by operation.

The bounds are those the operations are derived to: a reciprocal is off by half an ulp and
2^-17 (an integer Newton step on the rounded 43-bit seed, so the rounded reciprocal or
its neighbour), a reciprocal root by half an ulp and 2^-8; a root, one product more, is the
rounded root or its neighbour (2 x 0.504 + 1/2 ulps where the root's mantissa is near 2 and
the reciprocal's near 1), a ratio of roots off by half an ulp more at most; quotients and roots from an exact remainder are the rounded ones; conversions, powers of
two, signs and comparisons are exact."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import ec2d_build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
OPS = ("recip recip_any rroot root root_t root_ratio quot quot_any div_r sqrt_r to_float to_double twice half eighth neg "
       "below at_least above minmod tanh_pos sixth_root pos_part neg_part").split()
N = 1 << 21
LD = np.longdouble


@pytest.fixture(scope="module")
def op(tmp_path_factory, gpu_lib):
    so = str(tmp_path_factory.mktemp("arith") / "arith.so")
    subprocess.run([ec2d_build.nvcc(), *ec2d_build.ARCH, *ec2d_build.FLAGS, "-shared", "-I", ec2d_build.SRC,
                    os.path.join(HERE, "arith_probe.cu"), "-o", so, "-lcudart"], check=True, capture_output=True)
    fn = ctypes.CDLL(so).arith
    dp = ctypes.POINTER(ctypes.c_double)
    fn.argtypes = [ctypes.c_int, ctypes.c_longlong, dp, dp, dp]

    def call(name, a, b=None):
        a = np.ascontiguousarray(a, np.float64).ravel()
        b = np.ones_like(a) if b is None else np.ascontiguousarray(np.broadcast_to(b, a.shape), np.float64)
        out = np.empty_like(a)
        ptr = [x.ctypes.data_as(dp) for x in (a, b, out)]
        assert fn(OPS.index(name), a.size, *ptr) == 0
        return out
    return call


# mantissas at the edges of the seeds: powers of two and their neighbours, the ends of the
# words and of the bits that the float seeds are cut at
EDGE_BITS = np.unique(np.concatenate([
    np.array([0, 1, 2, (1 << 52) - 1, (1 << 52) - 2, (1 << 32) - 1, 1 << 32, (1 << 51), (1 << 51) - 1], np.uint64),
    np.array([1 << k for k in range(52)], np.uint64), np.array([(1 << 52) - (1 << k) for k in range(52)], np.uint64)]))


def _samples(seed, lo=-300, hi=300, signs=False):
    rng = np.random.default_rng(seed)
    m = rng.integers(0, 1 << 52, N, dtype=np.uint64)
    m[:EDGE_BITS.size * 8] = np.tile(EDGE_BITS, 8)
    x = np.ldexp((m | np.uint64(1023 << 52)).view(np.float64), rng.integers(lo, hi, N))
    x[:EDGE_BITS.size] = (EDGE_BITS | np.uint64(1023 << 52)).view(np.float64)
    x[EDGE_BITS.size:2 * EDGE_BITS.size] = 2.0 * x[:EDGE_BITS.size]  # (odd and even exponents)
    return x * rng.choice([-1.0, 1.0], N) if signs else x


def _ulps(out, exact):
    """largest error in ulps of the exact value"""
    if np.finfo(LD).nmant < 63:
        pytest.skip("no extended precision")
    r = np.abs(exact.astype(np.float64))
    return float(np.max(np.abs(out.astype(LD) - exact) / np.spacing(r)))


def test_reciprocals(op):
    x = _samples(1, -1021, 1021, signs=True)
    for name in ("recip", "recip_any"):
        assert _ulps(op(name, x), 1 / x.astype(LD)) <= 0.5 + 2.0 ** -16
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** 1022])
    assert np.all(np.isnan(op("recip", odd)))
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(op("recip_any", odd), 1.0 / odd)


def test_roots(op):
    x = _samples(2, -1021, 1021)
    s = np.sqrt(x.astype(LD))
    assert _ulps(op("rroot", x), 1 / s) <= 0.504
    for name in ("root", "root_t"):
        assert np.abs(op(name, x).view(np.int64) - np.sqrt(x).view(np.int64)).max() <= 1
    a, b = _samples(3), _samples(4)
    assert _ulps(op("root_ratio", a, b), np.sqrt(a.astype(LD) / b.astype(LD))) <= 2.01
    assert np.all(np.isnan(op("rroot", [0.0, -1.0, np.inf, np.nan])))
    np.testing.assert_array_equal(op("root", [0.0, -0.0]), [0.0, -0.0])
    assert np.all(np.isnan(op("root", [-1.0, np.nan])))
    with np.errstate(all="ignore"):
        odd = np.array([0.0, -0.0, -1.0, np.inf, np.nan])
        np.testing.assert_array_equal(op("root_t", odd), np.sqrt(odd))


def test_rounded_quotients_and_roots(op):
    a, b = _samples(5, signs=True), _samples(6, signs=True)
    for name in ("quot", "quot_any", "div_r"):
        np.testing.assert_array_equal(op(name, a, b), a / b)
    np.testing.assert_array_equal(op("sqrt_r", a[a > 0]), np.sqrt(a[a > 0]))
    with np.errstate(all="ignore"):
        odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e300, -1e300, 1e-310])
        for d in (3.0, -7e-5, 1e20):
            np.testing.assert_array_equal(op("quot_any", odd[:7], d), odd[:7] / d)
        d = np.array([0.0, np.inf, np.nan, -1e-300, 1e305, 5e-324])
        u, v = (x.ravel() for x in np.meshgrid(np.concatenate([odd, [1.0, 3.0]]), d))
        np.testing.assert_array_equal(op("div_r", u, v), u / v)
        np.testing.assert_array_equal(op("sqrt_r", np.concatenate([odd, d])), np.sqrt(np.concatenate([odd, d])))


def test_conversions(op):
    x = _samples(7, -160, 160, signs=True)
    # halfway between two floats, and its neighbours
    with np.errstate(over="ignore"):
        f = x[:1 << 18].astype(np.float32)
    f = f[np.isfinite(f) & (np.abs(f) > 1e-30) & (np.abs(f) < 1e30)]
    h = (f.astype(np.float64) + np.nextafter(f, np.float32(np.inf)).astype(np.float64)) / 2
    x = np.concatenate([x, h, np.nextafter(h, np.inf), np.nextafter(h, -np.inf),
                        [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-40, -1e-45, 1e-46, 2.0 ** -126, np.nextafter(2.0 ** -126, 0),
                         3.4028235677973366e38, 3.4028235677973362e38, 2.0 ** 127, 5e-324]])
    with np.errstate(all="ignore"):
        want = x.astype(np.float32)
    np.testing.assert_array_equal(op("to_float", x), want.astype(np.float64))
    np.testing.assert_array_equal(np.signbit(op("to_float", x[x == x])), np.signbit(x[x == x]))
    np.testing.assert_array_equal(op("to_double", want.astype(np.float64)), want.astype(np.float64))


def test_scalings_signs_and_comparisons(op):
    x = np.concatenate([_samples(8, -1015, 1020, signs=True), [0.0, -0.0, np.inf, -np.inf, np.nan]])
    for name, k in (("twice", 2.0), ("half", 0.5), ("eighth", 0.125)):
        np.testing.assert_array_equal(op(name, x), x * k)
    np.testing.assert_array_equal(op("neg", x), -x)
    np.testing.assert_array_equal(np.signbit(op("neg", [0.0, -0.0])), [True, False])
    num = x[x == x]
    np.testing.assert_array_equal(op("pos_part", num), np.where(np.signbit(num), 0.0, num))
    np.testing.assert_array_equal(op("neg_part", num), np.where(np.signbit(num), num, 0.0))
    y = np.abs(np.concatenate([_samples(9, -3, 3), [0.0, 1.0, 1.0, 2.0, 3.0]]))
    x = np.concatenate([_samples(10, -3, 3, signs=True), [0.0, np.nan, 1.0, np.inf, -np.inf]])
    x[:1000] = y[:1000]
    x[1000:2000] = np.nextafter(y[1000:2000], 0)
    x[2000:3000] = np.nextafter(y[2000:3000], 9)
    np.testing.assert_array_equal(op("below", x, y), x < y)
    np.testing.assert_array_equal(op("at_least", x, y), x >= y)
    np.testing.assert_array_equal(op("above", x, y), x > y)


def test_minmod(op):
    a, b = _samples(11, -3, 3, signs=True), _samples(12, -3, 3, signs=True)
    a[:4000], b[:2000] = 0.0, -0.0
    b[4000:8000] = a[4000:8000]
    b[8000:9000], a[9000:10000] = np.nan, np.nan
    with np.errstate(invalid="ignore"):
        want = np.where(a * b <= 0.0, 0.0, np.where(np.abs(a) <= np.abs(b), a, b))
    np.testing.assert_array_equal(op("minmod", a, b), want)


def test_wall_functions(op):
    x = np.concatenate([np.linspace(22.0, 700.0, 100001), np.linspace(0.0, 22.0, 100001), [np.inf]])
    np.testing.assert_allclose(op("tanh_pos", x), np.tanh(x), rtol=2.0 ** -51, atol=0)
    assert np.all(op("tanh_pos", x[:100001]) == 1.0)
    # (65 / b)^(1/6), b = g^6 + 64: one rounding of the result, and a sixth of those of 1/65, b/65
    # and the last two products of w^6, relative; elsewhere by the library's functions
    def err(b):
        exact = (LD(65) / b.astype(LD)) ** (LD(1) / 6)
        return float(np.max(np.abs(op("sixth_root", np.full_like(b, 65.0), b).astype(LD) / exact - 1)))
    if np.finfo(LD).nmant >= 63:
        b = 64.0 + np.abs(_samples(13, -60, 110))[:1 << 18]
        assert err(b) <= (1.0 + 4.0 / 6.0 + 0.01) * 2.0 ** -53
        assert err(10.0 ** np.linspace(37.0, 250.0, 4096)) <= 2.0 ** -51
