"""The FP64 passes' products, quotients and square roots in integer operations (wf_int64.cuh)
against IEEE arithmetic on the host, bit for bit: random significands, exact ties and their
neighbours, quotients and roots next to a representable number or to the middle of two, significands
of all ones and of one bit, all exponents that the passes admit and the widest that the functions do."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from weldformgpu_gb300 import build as B

pytestmark = pytest.mark.gpu

N = 1 << 19
HERE = os.path.dirname(os.path.abspath(__file__))
ONE = np.uint64(1) << np.uint64(52)
MASK = ONE - np.uint64(1)


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("int_arith") / "int_arith.so")
    subprocess.run([B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "-fmad=false", "-shared", "-Xcompiler",
                                          "-fPIC", "-o", so, os.path.join(HERE, "int_arith.cu")],
                   check=True)
    f = C.CDLL(so).int_arith
    f.argtypes = [C.c_int, C.c_long, C.c_void_p, C.c_void_p, C.c_void_p]

    def run(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ones_like(a) if b is None else np.ascontiguousarray(b, dtype=np.float64)
        assert a.shape == b.shape
        out = np.empty_like(a)
        assert f(op, a.size, a.ctypes.data, b.ctypes.data, out.ctypes.data) == 0
        return out
    return run


def _same(got, want, *operands):
    want = np.where(want == 0.0, 0.0, want)              # a zero result is +0
    bad = np.nonzero(got.view(np.uint64) != want.view(np.uint64))[0]
    assert bad.size == 0, (bad.size, [(float(o[bad[0]]).hex(), float(want[bad[0]]).hex(),
                                       float(got[bad[0]]).hex()) for o in operands])


def _number(rng, sig, e):
    """Doubles of the 53-bit integers sig with random signs and exponents of [-e, e]."""
    exp = rng.integers(-e, e + 1, sig.size)
    x = np.ldexp(sig.astype(np.float64), exp - 52)
    return np.where(rng.random(sig.size) < 0.5, -x, x)


def _sig(rng, n=N):
    return rng.integers(0, 1 << 52, n, dtype=np.uint64) | ONE


def _special(rng, n=N):
    """Significands of one bit, all ones, runs of ones and their neighbours."""
    k = rng.integers(0, 53, n).astype(np.uint64)
    j = rng.integers(0, 53, n).astype(np.uint64)
    one = np.uint64(1)
    pick = rng.integers(0, 5, n)
    s = np.select([pick == 0, pick == 1, pick == 2, pick == 3],
                  [ONE | (one << k), (ONE << one) - (one << k), ONE | ((one << k) - one),
                   ONE | ((one << k) + (one << j))], ONE + (rng.integers(0, 4, n).astype(np.uint64)))
    return (s & MASK) | ONE


def _inverse(a):
    """a^-1 mod 2^64 of odd a, by Newton's iteration."""
    x = a.copy()
    for _ in range(6):
        x = x * (np.uint64(2) - a * x)
    return x


# the exponents of a pair's values (2^+-120), and such that the result is just normal
RANGES = (0, 1, 120, 510)


@pytest.mark.parametrize("e", RANGES)
@pytest.mark.parametrize("kind", ["random", "special", "ties", "near_ties"])
def test_products(evaluate, kind, e):
    rng = np.random.default_rng([e, len(kind)])
    if kind == "random":
        sa, sb = _sig(rng), _sig(rng)
    elif kind == "special":
        sa, sb = _special(rng), np.where(rng.random(N) < 0.5, _special(rng), _sig(rng))
    elif kind == "ties":
        # odd numbers of 27 bits: their product has 53 bits or 54, and then ends in a half
        odd = [rng.integers(1 << 26, 1 << 27, N, dtype=np.uint64) | np.uint64(1) for _ in range(2)]
        sa, sb = (o << np.uint64(26) for o in odd)
        assert ((odd[0] * odd[1]) >> np.uint64(53)).astype(bool).mean() > 0.2
    else:
        # the product's low bits are a half of the last place, give or take a few units of 2^-105
        sa = _sig(rng) | np.uint64(1)
        half = np.where(rng.random(N) < 0.5, np.uint64(1) << np.uint64(51), np.uint64(1) << np.uint64(52))
        low = half + rng.integers(-3, 4, N).astype(np.uint64)
        sb = ((_inverse(sa) * low) & ((ONE << np.uint64(1)) - np.uint64(1))) | ONE
    a, b = _number(rng, sa, e), _number(rng, sb, e)
    _same(evaluate(0, a, b), a * b, a, b)


@pytest.mark.parametrize("e", RANGES)
@pytest.mark.parametrize("kind", ["random", "special", "neighbours", "middles", "close"])
def test_quotients(evaluate, kind, e):
    rng = np.random.default_rng([e, len(kind), 1])
    sb = _sig(rng)
    if kind == "random":
        sa = _sig(rng)
    elif kind == "special":
        sa, sb = _special(rng), np.where(rng.random(N) < 0.5, _special(rng), sb)
    elif kind == "close":                                # a and b a few units apart: quotients near 1
        sa = np.clip(sb.astype(np.int64) + rng.integers(-3, 4, N), 1 << 52, (1 << 53) - 1).astype(np.uint64)
    else:
        # a = q b rounded, give or take two units, with q a double or the middle of two
        q = rng.integers(1 << 52, 1 << 53, N).astype(object)
        if kind == "middles":
            q = 2 * q + 1
        p = q * sb.astype(object)
        bits = np.array([int(v).bit_length() for v in p])
        sa = np.array([(int(v) >> (int(n) - 53)) for v, n in zip(p, bits)], dtype=np.int64)
        sa = np.clip(sa + rng.integers(-2, 3, N), 1 << 52, (1 << 53) - 1).astype(np.uint64)
    a, b = _number(rng, sa, e), _number(rng, sb, e)
    _same(evaluate(1, a, b), a / b, a, b)


@pytest.mark.parametrize("e", (0, 1, 240, 1020))
@pytest.mark.parametrize("kind", ["random", "special", "squares", "middles"])
def test_square_roots(evaluate, kind, e):
    rng = np.random.default_rng([e, len(kind), 2])
    if kind == "random":
        x = np.abs(_number(rng, _sig(rng), e))
    elif kind == "special":
        x = np.abs(_number(rng, _special(rng), e))
    else:
        # k k or (k + 1/2)^2 rounded, give or take two units; k of 53 bits, or of 26 (exact squares)
        k = rng.integers(1 << 52, 1 << 53, N).astype(object)
        k[: N // 4] = rng.integers(1 << 25, 1 << 26, N // 4).astype(object)
        if kind == "middles":
            k = 2 * k + 1
        p = k * k
        bits = [int(v).bit_length() for v in p]
        odd = np.array([n & 1 for n in bits])            # keeps the parity of the exponent
        s = np.array([int(v) >> (n - 53) if n > 53 else int(v) << (53 - n) for v, n in zip(p, bits)],
                     dtype=np.int64)
        s = np.clip(s + rng.integers(-2, 3, N), 1 << 52, (1 << 53) - 1).astype(np.float64)
        x = np.ldexp(s, (1 - odd) + 2 * rng.integers(-e // 2, e // 2 + 1, N) - 52)
    x[:8] = [0.0, 1.0, 4.0, 2.0, np.nextafter(1.0, 0.0), np.nextafter(4.0, 0.0), np.nextafter(1.0, 2.0),
             2.0**-1022]
    _same(evaluate(2, x), np.sqrt(x), x)


def test_zeros(evaluate):
    x = np.array([0.0, -0.0, 1.5, -2.0**120])
    a, b = (m.ravel() for m in np.meshgrid(x, x))
    _same(evaluate(0, a, b), a * b, a, b)
    a, b = a[b != 0.0], b[b != 0.0]
    _same(evaluate(1, a, b), a / b, a, b)
