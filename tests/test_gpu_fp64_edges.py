"""The branch-free IEEE divisions and roots at their hard operands: mantissas
of all ones and next to it, next to one, roots and quotients that lie next to
the midpoint of two doubles (formed in integers), over the exponents."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
M = 1 << 52


@pytest.fixture(scope="module")
def differ(sed_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("edges") / "fp64_edges.so")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "fp64_edges.cu")], check=True)
    f = C.CDLL(so).fp64_edges
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]

    def run(a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        bad = np.zeros(4, np.uint64)
        assert f(a.ctypes.data, b.ctypes.data, a.size, bad.ctypes.data) == 0
        return {k: int(v) for k, v in zip(("division", "reciprocal", "root", "reciprocal root"), bad)}

    return run


def test_mantissas_of_ones_and_next_to_one(differ):
    """Every pair of the mantissas within 40 steps of 1 on either side, at even
    and odd exponents, and the all-ones mantissa at every exponent whose
    residuals have all their bits (2^-105 of the operand is no less than the
    smallest subnormal)."""
    near = [(2 * M - 1 - k) for k in range(40)] + [M + k for k in range(40)]
    m = np.array([k / M for k in near])
    a, b = np.meshgrid(m, m)
    for ea, eb in ((0, 0), (1, 0), (-1, 7), (90, -60), (-141, 100)):
        assert not any(differ(np.ldexp(a, ea).ravel(), np.ldexp(b, eb).ravel()).values()), (ea, eb)
    e = np.arange(-1074 + 105 + 1, 1000)
    x = np.ldexp((2 * M - 1) / M, e)
    for one in (1.0, 1.5, (2 * M - 1) / M):
        assert not any(differ(x, np.full(e.size, one)).values()), one
    # as divisors over the exponents, dividends a power of two
    assert not any(differ(np.ldexp(1.0, e // 2), np.ldexp((2 * M - 1) / M, e // 2)).values())


def _hard_roots():
    """a = m^2 + m - k, whose root lies (k + 1/4) / (2 m) below m + 1/2: m from
    m^2 + m = k modulo 2^52 or 2^53, so that a has 53 bits."""
    out = []
    for bits in (52, 53):
        for k in range(-3000, 3001, 2):
            for root in (0, 1):
                m = root
                for i in range(1, bits):
                    if (m * m + m - k) >> i & 1:
                        m |= 1 << i
                for x in ((m, m + M) if bits == 52 else (m,)):
                    a = x * x + x - k
                    if M <= x < 2 * M and int(float(a)) == a:
                        out.append(float(a))
    return np.array(out)


def test_roots_next_to_midpoints(differ):
    a = _hard_roots()
    assert a.size > 5000
    r = a[:200]  # CUDA's root is the rounded one: (2 root - 1)^2 < 4 a < (2 root + 1)^2
    for x in r:
        s, n = int(math.sqrt(x)), int(x)
        assert (2 * s - 1) ** 2 < 4 * n < (2 * s + 1) ** 2
    for e in (0, -104, -40, 60):
        bad = differ(np.ldexp(a, e), np.ones(a.size))
        assert not any(bad.values()), (e, bad)


def test_quotients_next_to_midpoints(differ):
    """a 2^54 = b q + r with q of 54 bits and odd: a / b lies r / b of half a
    unit from the midpoint of two doubles."""
    rng = np.random.default_rng(4)
    A, B = [], []
    for t in range(40000):
        b = (M | int(rng.integers(0, M)) | 1) if t % 5 else 2 * M - 1 - 2 * (t % 250)
        r = 2 * int(rng.integers(-20, 20)) + 1
        q = (-r * pow(b, -1, 1 << 54)) % (1 << 54)
        a, rest = divmod(b * q + r, 1 << 54)
        assert rest == 0 and q & 1
        if q >> 53 and M <= a < 2 * M:
            A.append(float(a))
            B.append(float(b))
    assert len(A) > 10000
    for ea, eb in ((0, 0), (-52, -52), (-90, 30)):
        bad = differ(np.ldexp(A, ea), np.ldexp(B, eb))
        assert bad["division"] == 0 and bad["reciprocal"] == 0, (ea, eb, bad)
