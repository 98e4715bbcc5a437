"""The branch-free division and square root of the step kernels (fcb_arith.cuh)
against the operators, bit for bit, where their flag says they hold; the flag
itself over the operands it must refuse."""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def check(gpu_lib, tmp_path_factory):
    so = tmp_path_factory.mktemp("arith") / "arith_check.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", "-I", str(ROOT / "forestclaw_b200" / "csrc"),
                    str(ROOT / "tests" / "arith_check.cu"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    dp, ip = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    lib.run_check.argtypes = [dp, dp, ctypes.c_int, dp, ip]

    def run(a, b):
        a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in (a, b))
        out, ok = np.empty((6, a.size)), np.empty((2, a.size), dtype=np.int32)
        rc = lib.run_check(a.ctypes.data_as(dp), b.ctypes.data_as(dp), a.size, out.ctypes.data_as(dp),
                           ok.ctypes.data_as(ip))
        assert rc == 0
        return out, ok.astype(bool)

    return run


def _mantissas(g, n):
    return g.integers(1 << 52, 1 << 53, n).astype(np.float64)


def test_random_operands(check):
    """Mantissas at random, exponents over the whole accepted range."""
    g = np.random.default_rng(0)
    n = 1 << 21
    a = np.ldexp(_mantissas(g, n), g.integers(-1000, 40, n)) * g.choice([-1.0, 1.0], n)
    b = np.ldexp(_mantissas(g, n), g.integers(-950, 6, n))
    out, ok = check(a, b)
    assert ok.mean() > 0.9
    both = ok[0] & (np.abs(out[1]) < 1e300) & (np.abs(out[1]) > 1e-300)
    assert np.array_equal(out[0][both], out[1][both])
    assert np.array_equal(out[2][ok[1]], out[3][ok[1]])


def test_quotients_next_to_the_middle_of_two_doubles(check):
    """a is the double nearest to m b for a midpoint m of two doubles (and its
    neighbours): the quotients that are hardest to round.  Divisors include
    mantissas next to 1 and 2."""
    g = np.random.default_rng(1)
    n = 60000
    mid = 2 * g.integers(1 << 52, 1 << 53, n) + 1  # 54 bits, odd
    b = g.integers(1 << 52, 1 << 53, n)
    b[:64] = (1 << 53) - 1 - np.arange(64)
    b[64:128] = (1 << 52) + np.arange(64)
    a = np.array([float(int(m) * int(d)) for m, d in zip(mid, b)])
    a = np.concatenate([a, np.nextafter(a, np.inf), np.nextafter(a, 0)])
    bb = np.tile(b.astype(np.float64), 3)
    out, ok = check(np.ldexp(a, -107), np.ldexp(bb, -52))
    assert ok[0].all()
    assert np.array_equal(out[0], out[1])


def test_reciprocals(check):
    """Powers of two over divisors next to powers of two, all ones included (the
    speed of a depth one rounding below 1), and over random ones."""
    g = np.random.default_rng(4)
    k = np.arange(1, 200)
    b = np.concatenate([1.0 - k * 2.0 ** -53, 1.0 + k * 2.0 ** -52, np.ldexp(_mantissas(g, 1 << 20), -52)])
    for a in (0.5, 1.0, -2.0 ** -200):
        for scale in (1.0, 2.0 ** 7, 2.0 ** -800):
            out, ok = check(np.full_like(b, a), b * scale)
            assert ok[0].all()
            assert np.array_equal(out[0], out[1])


def test_square_roots_next_to_the_middle_of_two_doubles(check):
    """x next to the square of a midpoint: random ones, and the closest there are
    (m^2 = j mod 2^k for small j, lifted bit by bit)."""
    g = np.random.default_rng(2)
    xs = []
    for m in g.integers(1 << 52, 1 << 53, 40000):
        sq = (2 * int(m) + 1) ** 2
        for k in (52, 53):
            x = float(sq >> k)
            xs += [x, np.nextafter(x, 0), np.nextafter(x, np.inf)]
    for j in range(1, 8 * 400, 8):
        for k in (54, 55):
            r = 1
            for bit in range(3, k + 1):  # r^2 = j mod 2^bit
                if (r * r - j) % (1 << bit):
                    r += 1 << (bit - 2)
            for root in (r, (1 << k) - r, r + (1 << (k - 1)), (1 << (k - 1)) - r):
                root %= 1 << k
                if root.bit_length() == 54 and (root * root - j) % (1 << 53) == 0:
                    xs.append(float((root * root - j) >> 53))
                    xs.append(2.0 * xs[-1])
    x = np.array(xs)
    x = np.concatenate([np.ldexp(x, -53), np.ldexp(x, -54), np.ldexp(x, -700)])
    out, ok = check(np.ones_like(x), x)
    assert ok[1].all()
    assert np.array_equal(out[2], out[3])


def test_quotients_by_pi(check):
    g = np.random.default_rng(3)
    n = 1 << 20
    a = np.concatenate([np.ldexp(_mantissas(g, n), g.integers(-800, -50, n)), [0.0, 1.0, 3.141592653589793]])
    out, _ = check(a, np.ones_like(a))
    assert np.array_equal(out[4], out[5])


def test_operands_the_flag_refuses(check):
    tiny, inf, nan = 5e-324, np.inf, np.nan
    b = np.array([0.0, -0.0, tiny, 1e-300, 1e30, inf, nan, -1.0])
    _, ok = check(np.ones_like(b), b)
    assert not ok[0].any()
    _, ok = check(np.ones(6), np.array([0.0, tiny, 1e-300, -1.0, inf, nan]))
    assert not ok[1].any()
    a = np.array([1e-300, -1e-300, 2.0 ** -1000])
    _, ok = check(a, np.ones_like(a))
    assert not ok[0].any()
    out, ok = check(np.array([0.0, -0.0]), np.array([3.0, 3.0]))
    assert ok[0].all() and (out[0] == 0).all()


def test_dividends_the_flag_refuses(check):
    """Infinite, NaN and huge dividends: the operator's infinity, not the residual's NaN."""
    a = np.array([np.inf, -np.inf, np.nan, 1e300, -1e300, 1.7e308, 2.0 ** 123])
    for b in (1.0, 1e-250, 3.0):
        _, ok = check(a, np.full_like(a, b))
        assert not ok[0].any()
    a = np.array([np.nextafter(2.0 ** 123, 0), -1e37, 2.0 ** -960, -(2.0 ** -960)])
    for b in (2.0 ** -900, 0.7, 2.0 ** 59 * 1.3):
        out, ok = check(a, np.full_like(a, b))
        assert ok[0].all()
        big = np.abs(out[1]) >= 2.0 ** -1022
        assert np.isfinite(out[1]).all() and np.array_equal(out[0][big], out[1][big])
