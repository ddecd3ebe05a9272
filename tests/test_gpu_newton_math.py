"""The branch-free FP64 reciprocal, quotient and square root of the face states
against CUDA's operators (and the CPU's): wherever they accept their operands
they give the same bits, and they accept what a run's states hold."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from raishinsource_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def newton(tmp_path_factory):
    """newton(a, b) -> (out[6, n], ok[3, n])"""
    so = str(tmp_path_factory.mktemp("newton") / "newton_math.so")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", *build.ARCH, "--fmad=true", "-shared", "-Xcompiler", "-fPIC",
                    "-o", so, os.path.join(HERE, "newton_math.cu")], check=True)
    f = C.CDLL(so).newton_math
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]

    def call(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        out, ok = np.empty((6, a.size)), np.empty(a.size, np.int32)
        assert f(a.ctypes.data, b.ctypes.data, a.size, out.ctypes.data, ok.ctypes.data) == 0
        return out, np.array([(ok >> k) & 1 for k in range(3)], bool)
    return call


def make(sig, exp):
    """sig: 52-bit fractions, exp: unbiased exponents."""
    return (sig.astype(np.uint64) | ((exp + 1023).astype(np.uint64) << np.uint64(52))).view(np.float64)


def hard(rng, n):
    """Operand pairs (a, b), b > 0: random ones over the whole accepted range,
    significands next to one, to two and to a power of two's neighbours, quotients and
    square roots next to the middle between two doubles."""
    top = 1 << 52
    sig = [rng.integers(0, top, (2, n), dtype=np.uint64)]
    near = rng.integers(0, 64, (2, n), dtype=np.uint64)
    sig.append(near)
    sig.append(np.uint64(top - 1) - near)
    sig.append(np.uint64(1) << rng.integers(0, 52, (2, n)).astype(np.uint64))
    a, b = [], []
    for s in sig:
        a.append(make(s[0], rng.integers(-500, 500, n)))
        b.append(make(s[1], rng.integers(-500, 500, n)))
    # a = (q + half an ulp) b to one rounding, and its neighbours
    q, d = make(rng.integers(0, top, n, dtype=np.uint64), np.zeros(n, int)), make(sig[0][1], np.zeros(n, int))
    m = ((q.astype(np.longdouble) + np.longdouble(2.0 ** -53)) * d.astype(np.longdouble)).astype(np.float64)
    # b = (g + half an ulp)^2 to one rounding, and its neighbours
    h = ((q.astype(np.longdouble) + np.longdouble(2.0 ** -53)) ** 2).astype(np.float64)
    for k in (-np.inf, np.inf):
        a += [np.nextafter(m, k), m]
        b += [d, np.nextafter(h, k)]
    a.append(m)
    b.append(h)
    a = np.concatenate(a)
    return a * np.where(rng.random(a.size) < 0.5, -1.0, 1.0), np.concatenate(b)


def test_same_bits_as_the_operators(newton):
    rng = np.random.default_rng(5)
    for _ in range(8):
        a, b = hard(rng, 1 << 18)
        out, ok = newton(a, b)
        want = np.array([1.0 / b, a / b, np.sqrt(b)])
        for k in range(3):
            assert np.array_equal(out[3 + k], want[k])  # the operators are IEEE's
            assert np.array_equal(out[k][ok[k]], want[k][ok[k]])
        low = (b.view(np.uint64) & np.uint64(0xffffffff)) == np.uint64(0xffffffff)  # refused as a divisor
        assert low.any()
        assert np.array_equal(ok[0], ~low) and np.array_equal(ok[1], ~low) and ok[2].all()


@pytest.mark.parametrize("bad", [0.0, -0.0, 2.0 ** -501, 2.0 ** 500, 5e-324, np.inf, -np.inf, np.nan,
                                 1.0 - 2.0 ** -53, 2.0 - 2.0 ** -52])
def test_operands_that_are_refused(newton, bad):
    """As a divisor; as a numerator or radicand a significand of all ones is in order."""
    out, ok = newton(np.ones(1), np.array([bad]))
    ones = abs(bad) in (1.0 - 2.0 ** -53, 2.0 - 2.0 ** -52)
    assert not ok[0] and not ok[1] and ok[2] == ones
    out, ok = newton(np.array([bad]), np.array([3.0]))
    assert ok[0] and ok[1] == ones


def test_operands_at_the_ends_of_the_range(newton):
    b = np.array([2.0 ** -500, np.nextafter(2.0 ** 500, 0.0) * (1 - 2.0 ** -52), 1.0, np.nextafter(1.0, 2.0)])
    a = b[::-1].copy()
    out, ok = newton(a, b)
    assert ok.all()
    assert np.array_equal(out[:3], out[3:])
