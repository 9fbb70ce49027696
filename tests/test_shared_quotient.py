"""The FP64 pair code's shared quotient (x r corrected once by its remainder, r = 1/y rounded)
is the correctly rounded x / y: the argument beside the code, checked in exact arithmetic over
all mantissas of small formats and at its three hard pairs in FP64, and the device function
against the device's division."""
from __future__ import annotations

import ctypes
import os
import subprocess
from fractions import Fraction as F

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _round(v: F, p: int) -> F:
    """v to p significant bits, ties to even."""
    if v == 0:
        return v
    s, v = (-1, -v) if v < 0 else (1, v)
    e = v.numerator.bit_length() - v.denominator.bit_length()
    if F(2) ** e > v:
        e -= 1
    ulp = F(2) ** (e - p + 1)
    k, rest = divmod(v, ulp)
    k += rest * 2 > ulp or (rest * 2 == ulp and k % 2)
    return s * k * ulp


def _quotient(x: F, y: F, p: int) -> F:
    r = _round(1 / y, p)
    q = _round(x * r, p)
    return _round(q + _round(x - y * q, p) * r, p)


@pytest.mark.parametrize("p", [3, 4, 5, 6, 7])
def test_all_mantissas_of_small_formats(p):
    one = 1 << (p - 1)
    for i in range(one, 2 * one):
        for j in range(one, 2 * one):
            x, y = F(i, one), F(j, one)
            assert _quotient(x, y, p) == _round(x / y, p), (i, j)


def test_the_hard_pairs_of_fp64():
    u = F(2) ** -52
    for m in range(1, 5):
        for n in range(1, 5):
            x, y = 2 - m * u, 2 - n * u
            assert _quotient(x, y, 53) == _round(x / y, 53), (m, n)


@pytest.mark.gpu
def test_device_quotients(library, tmp_path):
    from spherocyls_gb300 import build

    so = os.path.join(str(tmp_path), "libquotient_probe.so")
    subprocess.run([os.path.join(build.cuda_home(), "bin", "nvcc"), *build.ARCH, "-O3",
                    "-std=c++17", "-fmad=false", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "quotient_probe.cu"), f"-I{build.CSRC}"], check=True)
    lib = ctypes.CDLL(so)
    rng = np.random.default_rng(7)
    n = 1 << 22

    def mantissas(k):
        """Random ones, ones near 1 and 2, short ones (quotients near midpoints)."""
        kind = rng.integers(0, 4, k)
        m = rng.integers(1 << 52, 1 << 53, k)
        near = rng.integers(0, 8, k)
        m = np.where(kind == 1, (1 << 52) + near, m)
        m = np.where(kind == 2, (1 << 53) - 1 - near, m)
        m = np.where(kind == 3, (m >> 27) << 27, m)
        return m.astype(np.float64)

    # divisors over the whole range (past 2^+-500 a division), dividends within it
    x = np.ldexp(mantissas(n) * rng.choice([-1.0, 1.0], n), rng.integers(-540, 440, n))
    y = np.ldexp(mantissas(n), rng.integers(-1120, 960, n))
    # dividends made from a quotient next to a midpoint, where rounding is hardest
    h = n // 2
    q = mantissas(h) + 0.5 * rng.integers(-1, 2, h)
    y[:h] = np.ldexp(mantissas(h), -52)
    x[:h] = np.ldexp(q, -52) * y[:h]
    out = np.full(n, -1, dtype=np.int32)
    ptr = lambda a, t: a.ctypes.data_as(ctypes.POINTER(t))
    assert lib.probe_quotients(ptr(x, ctypes.c_double), ptr(y, ctypes.c_double), n,
                               ptr(out, ctypes.c_int)) == 0
    assert not out.any()
