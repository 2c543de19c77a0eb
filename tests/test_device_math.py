"""The arithmetic that stands in for FP64 in the FP32 kernels, function by
function on the GPU over its whole range, against integers or numpy's long
double; and the index arithmetic of the time unfolding.

The bounds follow from the operations (u = 2^-24, a float's rounding):
df_div2      the first digit is within 2^-22 of the quotient, the second as near
             to the remainder: 2^-44, plus the roundings of the remainder: 2^-43;
1 - sqrt     x / 2 + x^2 / 8 in pairs (2^-46 each) and a rest below 6e-7 of the
             value within 8 u: 2^-41.7 + 2^-44; through df_sqrt and df_div 2^-44;
(1-x)^(3/2)  the rest is below 1.6e-6 within 8 u: 2^-40.3, plus 2^-45;
df_split     29 low bits rounded to 24: 2^-48 (conversions: 2^-48, below float's
             range half its smallest step);
norm32       two exact products, their errors added: 4 u^2 = 2^-46, and what a
             component 2^-63 of the other loses;
ln32         e ln 2, the table and r, r^2 / 2 added in pairs, 2^-46 of the largest
             partial sum each: 3 2^-46 max(1, |ln|), the rest in float: 2^-43;
cis_turn     CUDA's stated bound of __sinf / __cosf in [-pi, pi], 2^-21.19, and
             the angle's rounding, pi u: 7e-7.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def dm(lib_path, tmp_path_factory):
    from sentinel1_decode_gb300.build import ARCH, SRC, nvcc
    so = str(tmp_path_factory.mktemp("device_math") / "device_math.so")
    out = os.path.dirname(lib_path)
    subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", SRC,
                    os.path.join(HERE, "device_math", "device_math.cu"), "-o", so, "-L", out, "-ls1g",
                    "-Xlinker", "-rpath=" + out], check=True)
    lib = ctypes.CDLL(so)

    def call(name, *args):
        getattr(lib, "dm_" + name)(*[a.ctypes.data_as(ctypes.c_void_p) if isinstance(a, np.ndarray) else ctypes.c_int(a)
                                     for a in args])
    return call


N = 1 << 18


def spread(rng, lo, hi, n=N):
    """Values over the range, even in their logarithm."""
    return np.exp2(rng.uniform(np.log2(lo), np.log2(hi), n)) * rng.uniform(1, 1.0000001, n)


def test_quotient(dm):
    rng = np.random.default_rng(1)
    x = spread(rng, 2.0 ** -40, 2.0 ** 40) * rng.choice([-1, 1], N)
    y = spread(rng, 2.0 ** -30, 2.0 ** 30) * rng.choice([-1, 1], N)
    out = np.zeros(N)
    dm("pairs", 0, x, y, out, N)
    want = x.astype(np.longdouble) / y
    assert float(np.max(np.abs(out - want) / np.abs(want))) < 2.0 ** -43


@pytest.mark.parametrize("what", [1, 2])
def test_squint_series(dm, what):
    """x over the whole of it, the line between series and roots (2e-3) included."""
    rng = np.random.default_rng(2)
    x = np.concatenate([spread(rng, 1e-12, 0.5), spread(rng, 1.999e-3, 2.001e-3), [0.0]])
    n = x.size
    y, out = np.ones(n), np.zeros(n)
    dm("pairs", what, x, y, out, n)
    x = x.astype(np.longdouble)
    r = np.sqrt(1 - x)
    want = x / (1 + r) if what == 1 else r * r * r
    err = np.abs(out - want)[:-1] / np.abs(want)[:-1]
    assert float(err.max()) < (2.0 ** -41 if what == 1 else 2.0 ** -40)
    assert out[-1] == (0.0 if what == 1 else 1.0)


def test_split(dm):
    rng = np.random.default_rng(3)
    x = np.concatenate([spread(rng, 2.0 ** -62, 2.0 ** 127) * rng.choice([-1, 1], N), spread(rng, 1e-44, 2.0 ** -61),
                        [0.0, 2.0 ** -62, -2.0 ** 126, 1.0, -1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0)]])
    n = x.size
    out = np.zeros((n, 2))
    dm("split", x, out, n)
    got = out[:, 0].astype(np.longdouble) + out[:, 1]
    big = np.abs(x) >= 2.0 ** -62
    assert float(np.max(np.abs(got - x)[big] / np.abs(x)[big])) <= 2.0 ** -48
    assert float(np.max(np.abs(got - x)[~big] - 2.0 ** -48 * np.abs(x)[~big])) <= 2.0 ** -150
    assert np.array_equal(out.astype(np.float32), out)


def test_norm_and_logarithm(dm):
    """Every size of a float, subnormal and largest ones included, components alike
    and far apart, and magnitudes next to 1 where the logarithm vanishes."""
    rng = np.random.default_rng(4)
    a = spread(rng, 2.0 ** -148, 1.9999 * 2.0 ** 126)
    b = a * np.exp2(-rng.uniform(0, 30, N))
    v = np.stack([a, np.where(rng.random(N) < 0.1, 0, b)], 1)
    one = 1 + np.exp2(-rng.uniform(1, 24, 4096))[:, None] * np.array([1.0, 0.0]) - np.array([0.0, 1.0])
    edge = [[np.finfo(np.float32).max] * 2, [2.0 ** -149, 0], [2.0 ** -64, 0], [2.0 ** -64 * (1 - 2.0 ** -24), 0],
            [1, 0], [0, 1], [1, 1], [2.0 ** 127, 0]]
    v = np.concatenate([v, v[:, ::-1], one, edge]).astype(np.float32)
    v = v[np.abs(v).max(1) > 0]
    v *= rng.choice([-1, 1], v.shape).astype(np.float32)
    n = len(v)
    out, e = np.zeros((n, 4)), np.zeros(n, np.int32)
    dm("norm_log", np.ascontiguousarray(v), out, e, n)
    w = np.ldexp(v.astype(np.longdouble), -e[:, None])
    norm = (w * w).sum(1)
    got = out[:, 0].astype(np.longdouble) + out[:, 1]
    assert out[:, 0].min() >= 1 and out[:, 0].max() < 32
    assert float(np.max(np.abs(got - norm) / norm)) < 2.0 ** -45
    ln = np.log(norm) + 2 * e * np.log(np.longdouble(2))
    err = np.abs(out[:, 2].astype(np.longdouble) + out[:, 3] - ln)
    assert float(np.max(err / (3 * 2.0 ** -46 * np.maximum(1, np.abs(ln)) + 2.0 ** -43))) < 1


def test_norm_of_nothing(dm):
    v, out, e = np.zeros((3, 2), np.float32), np.zeros((3, 4)), np.zeros(3, np.int32)
    v[1, 1] = np.nan
    v[2, 0] = np.inf
    dm("norm_log", v, out, e, 3)
    assert out[0, 0] == 0 and out[0, 1] == 0
    assert not np.isfinite(out[1:, 0]).any()


def test_phase_factor(dm):
    rng = np.random.default_rng(5)
    hi = np.concatenate([rng.uniform(-0.5, 0.5, N), [0, 0.25, -0.25, 0.5, -0.5]]).astype(np.float32)
    lo = (rng.uniform(-1, 1, hi.size) * 2.0 ** -25 * np.abs(hi)).astype(np.float32)
    t, out = np.stack([hi, lo], 1), np.zeros((hi.size, 2), np.float32)
    dm("cis", t, out, hi.size)
    ang = 2 * np.arccos(np.longdouble(-1)) * (hi.astype(np.longdouble) + lo)
    err = np.hypot(out[:, 0] - np.cos(ang), out[:, 1] - np.sin(ang))
    assert float(err.max()) < np.sqrt(2) * 7e-7


@pytest.mark.parametrize("S,T,M", [(8, 1, 64), (61, 2, 96), (1201, 9, 960), (6908, 6, 10240), (13801, 3, 8192), (26700, 64, 24576)])
def test_axes_of_the_time_unfolding(dm, S, T, M):
    TS = S * T
    rng = np.random.default_rng(6)
    u = np.arange(TS) if TS < N else np.unique(np.concatenate([rng.integers(0, TS, N), [0, 1, TS - 2, TS - 1]]))
    u = u.astype(np.int32)
    out = np.zeros((u.size, 4), np.int32)
    dm("index", u, out, u.size, S, TS, 2 * M)
    u = u.astype(np.int64)
    iv = np.minimum(u * (S - 1) // (TS - 1), S - 2)
    first = -(-iv * (TS - 1) // (S - 1))
    np.testing.assert_array_equal(out[:, 0], iv)
    np.testing.assert_array_equal(out[:, 1], u - first)
    np.testing.assert_array_equal(out[:, 2], first)
    np.testing.assert_array_equal(out[:, 3], -(-(u % (2 * M) - 13) * TS // (2 * M)))
