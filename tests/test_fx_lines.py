"""Fixed-point line derivatives (csrc/fx.cuh) on the host, against the
derivative summed in long double.

The spectral second derivative of a line is a circulant sum with the kernel
c_j = -(1/N) sum_k f_k^2 cos(2 pi j k / N) (laplacian_3d's multiplier along one
axis, Pseudospec/openmp_dev/fftw_mod.f90:192-201).  Its error is compared with
that of the FP64 transform of the same line (numpy) and with a bound: the line
enters with an error below 2^-53 of its largest deviation, the multiplier
(2 f / N)^2 <= 1 does not amplify it, so the result is within a few 2^-53 of
(N/2)^2 max|x - x_0|.  Built with the undefined-behaviour sanitizer's trap, a
signed overflow anywhere ends the process.
"""
from __future__ import annotations

import ctypes as C
import functools
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
SIZES = [16, 32, 64, 128, 256, 512]
PADDED = [9, 10, 17, 32, 33, 64, 65, 96, 128, 129, 150, 251, 256]  # run on 64 ... 512 points


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    so = tmp_path_factory.mktemp("fx") / "libfx.so"
    subprocess.run(["g++", "-O1", "-std=gnu++17", "-shared", "-fPIC", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-o", str(so), str(HERE / "fx_lines.cpp")], check=True)
    lib = C.CDLL(str(so))
    dp = C.POINTER(C.c_double)
    lib.fx_line.argtypes = [C.c_int, C.c_int, dp, C.c_double, dp]
    lib.fx_round.argtypes = [C.c_longlong]
    lib.fx_round.restype = C.c_double

    def line(a, b, dk2=1.0, padded=False):
        n = len(a)
        m = max(64, 1 << (2 * n - 2).bit_length()) if padded else n
        x = np.ascontiguousarray(np.stack([a, b]), np.float64)
        out = np.empty_like(x)
        assert lib.fx_line(n, m, x.ctypes.data_as(dp), dk2, out.ctypes.data_as(dp)) == 0
        return out
    line.round = lib.fx_round
    return line


def kernel(n):
    f = np.minimum(np.arange(n), n - np.arange(n)).astype(np.longdouble)
    j = np.arange(n)
    # 8 atan(1): 2 pi in the platform's long double
    ang = 8 * np.arctan(np.longdouble(1)) * (np.outer(j, j) % n).astype(np.longdouble) / n
    return -(np.cos(ang) * f * f).sum(1) / n


def exact(x, c):
    n = len(x)
    i = np.arange(n)
    d = x.astype(np.longdouble) - np.longdouble(x[0])  # the kernel does not see a constant
    return c[(i[:, None] - i[None, :]) % n] @ d


def fp64(a, b):
    n = len(a)
    f = np.minimum(np.arange(n), n - np.arange(n)).astype(float)
    z = np.fft.ifft(-(f * f) * np.fft.fft((a - a[0]) + 1j * (b - b[0])))
    return z.real, z.imag


def inputs(n, kind, rng):
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    i = np.arange(n)
    if kind == "mean":  # a fluctuation on a large constant
        return 1.0 + 1e-5 * a, -300.0 + 1e-3 * b
    if kind == "smooth":
        k = np.arange(1, max(2, n // 4))
        ph = rng.uniform(0, 6.28, (2, len(k)))
        s = [(np.cos(2 * np.pi * np.outer(i, k) / n + p) / k ** 2).sum(1) for p in ph]
        return s[0], s[1]
    if kind == "spike":
        s = 1e-6 * a
        s[n // 3] = 1.0
        return s, b
    if kind == "nyquist":  # the largest derivative a line of its size can have
        return np.where(i % 2, 1.0, -1.0), np.where(i % 2, -1.0, 1.0)
    if kind == "aligned":  # every term of one spectral sum adds up
        k = 3
        return np.sign(np.cos(2 * np.pi * k * i / n) + 1e-9), np.sign(np.sin(2 * np.pi * k * i / n) + 1e-9)
    if kind == "uneven":
        return a, 1e-12 * b
    if kind == "tiny":
        return 1e-290 * a, 1e-280 * b
    if kind == "large":
        return 1e290 * a, b
    return a, b


@pytest.mark.parametrize("kind", ["noise", "mean", "smooth", "spike", "nyquist", "aligned", "uneven", "tiny", "large"])
@pytest.mark.parametrize("n,padded", [(n, False) for n in SIZES] + [(n, True) for n in PADDED])
def test_line_against_long_double(fx, n, padded, kind):
    rng = np.random.default_rng(n)
    c = kernel(n)
    worst = np.zeros(2)
    for _ in range(4):
        a, b = inputs(n, kind, rng)
        out = fx(a, b, padded=padded)
        ref64 = fp64(a, b)
        for l, x in enumerate((a, b)):
            e = exact(x, c)
            top = float(np.max(np.abs(x - x[0]))) * (n / 2) ** 2
            assert np.max(np.abs(out[l] - e)) <= 8 * 2.0 ** -53 * top
            norm = np.sqrt(np.sum(e * e))
            if l == 0 or kind not in ("uneven", "tiny", "large"):  # the FP64 transform mixes the two lines
                worst += [float(np.sqrt(np.sum((out[l] - e) ** 2)) / norm),
                          float(np.sqrt(np.sum((ref64[l] - e) ** 2)) / norm)]
    # no further off than the FP64 transform of the same line (both errors may
    # also be down to the rounding of the result itself, 2^-53)
    assert worst[0] <= 1.1 * worst[1] + 8 * 2.0 ** -53


@pytest.mark.parametrize("kind", ["uneven", "tiny", "large"])
@pytest.mark.parametrize("n,padded", [(n, False) for n in SIZES] + [(n, True) for n in PADDED])
def test_either_line_of_an_uneven_pair(fx, n, padded, kind):
    """Each line of a pair of very different size, against the FP64 transform of that line alone: its own
    exponent keeps it as exact as a line of a like pair."""
    rng = np.random.default_rng(100 + n)
    c = kernel(n)
    worst = np.zeros((2, 2))
    for _ in range(4):
        pair = inputs(n, kind, rng)
        out = fx(*pair, padded=padded)
        for l, x in enumerate(pair):
            e = exact(x, c)
            norm = np.sqrt(np.sum(e * e))
            alone = fp64(x, np.zeros(n))[0]
            worst[l] += [float(np.sqrt(np.sum((v - e) ** 2)) / norm) for v in (out[l], alone)]
    for l in (0, 1):
        assert worst[l][0] <= 1.1 * worst[l][1] + 8 * 2.0 ** -53, l


@pytest.mark.parametrize("n,padded", [(n, False) for n in SIZES] + [(n, True) for n in PADDED])
def test_line_special_values(fx, n, padded):
    fx = functools.partial(fx, padded=padded)
    z = np.zeros(n)
    assert np.array_equal(fx(z, z), np.zeros((2, n)))
    c = np.full(n, -0.7)
    assert np.array_equal(fx(c, c), np.zeros((2, n)))  # a constant has no derivative, exactly
    x = np.random.default_rng(0).standard_normal(n)
    keep = fx(x, c)
    for v in (np.nan, np.inf, -np.inf):
        y = x.copy()
        y[n // 2] = v
        out = fx(y, c)
        assert np.all(np.isnan(out[0])) and np.array_equal(out[1], keep[1])  # its own line only
    s = fx(np.where(np.arange(n) == 1, 5e-324, 0.0), x)  # subnormal values are not lost
    assert np.all(np.isfinite(s)) and s[0][1] < 0


def test_integer_to_double(fx):
    rng = np.random.default_rng(1)
    vals = [0, 1, -1, 2 ** 53, 2 ** 53 + 1, -(2 ** 53) - 3, 2 ** 62, -(2 ** 62), 2 ** 63 - 1, -(2 ** 63) + 1]
    vals += [int(v) >> int(s) for v, s in zip(rng.integers(-2 ** 63 + 1, 2 ** 63 - 1, 400), rng.integers(0, 63, 400))]
    for v in vals:
        got = fx.round(v) * 2.0 ** 61
        assert abs(int(got) - v) <= max(0, 2 ** (abs(v).bit_length() - 54))  # half a unit of the 53-bit result
