"""The quad kernels' arithmetic (ifosb_quad.cuh, ifosb_corr.cuh, k_dft's rounding) against
the plain operators, bit for bit: quotients from subnormal to overflowing, ties and near
ties of subnormal results, special operands, divisors outside the fast range, and products
whose sum must not be contracted. Seeded operands; no tolerance."""
import ctypes as C
import os

import numpy as np
import pytest

import ifosb

pytestmark = pytest.mark.gpu
N = 1 << 20
QUAD, TRIPLE, PRODUCT, BY_H, BY_POW2 = range(5)


@pytest.fixture(scope="module")
def check(ifosb_mod):
    so = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(ifosb.__file__))), "lib", "libquad_check.so")
    return C.CDLL(so)


def floats(rng, lo, hi, n=N):
    """Random signs and significands, exponents uniform in [lo, hi]; below -126: subnormals."""
    m = 1.0 + rng.integers(0, 1 << 23, n) / float(1 << 23)
    return (rng.choice([-1.0, 1.0], n) * m * np.exp2(rng.integers(lo, hi + 1, n).astype(np.float64))).astype(np.float32)


def with_special(rng, a):
    """Zeros of both signs, infinities and NaN in a sixteenth of the places."""
    at = rng.integers(0, len(a), len(a) // 16)
    a[at] = rng.choice(np.array([0.0, -0.0, np.inf, -np.inf, np.nan], np.float32), len(at))
    return a


def ties(rng, off):
    """a / b half-way between two subnormals, moved by `off` places of a."""
    odd = 2 * rng.integers(0, 1 << 9, N) + 1
    s = rng.integers(1, 15, N)
    b = (odd * np.exp2(s.astype(np.float64))).astype(np.float32)
    a = ((2 * rng.integers(0, 1 << 12, N) + 1) * odd * np.exp2((s - 150).astype(np.float64))).astype(np.float32)
    for _ in range(abs(off)):
        a = np.nextafter(a, np.float32(np.inf if off > 0 else 0), dtype=np.float32)
    return np.where(rng.integers(0, 2, N) == 1, a, -a).astype(np.float32), b


def run(check, what, a, b, in_range):
    a, b = (np.ascontiguousarray(x, np.float32) for x in (a, b))
    assert a.size == b.size and a.size % 4 == 0
    res = (C.c_int * 2)()
    ptr = lambda x: x.ctypes.data_as(C.c_void_p)
    assert check.quad_check(what, ptr(a), ptr(b), a.size, in_range, res) == 0
    q = min(res[1], a.size - 1)
    assert res[0] == 0, f"{res[0]} differ, first {a[q]!r} and {b[q]!r}"


@pytest.mark.parametrize("what", [QUAD, TRIPLE])
@pytest.mark.parametrize("lo,hi", [(-149, -110), (-130, -60), (-60, 60), (40, 127), (-149, 127)])
def test_division_in_range(check, what, lo, hi):
    rng = np.random.default_rng(lo + 3 * hi + 1000)
    b = np.abs(floats(rng, -10, 23))
    run(check, what, floats(rng, lo, hi), b, 1)
    run(check, what, with_special(rng, floats(rng, lo, hi)), b, 1)


@pytest.mark.parametrize("what", [QUAD, TRIPLE])
@pytest.mark.parametrize("off", [0, -1, 1, 2])
def test_division_on_ties_of_subnormals(check, what, off):
    run(check, what, *ties(np.random.default_rng(off + 9), off), 1)


@pytest.mark.parametrize("what", [QUAD, TRIPLE])
def test_division_by_anything(check, what):
    rng = np.random.default_rng(5)
    run(check, what, with_special(rng, floats(rng, -149, 127)), with_special(rng, floats(rng, -149, 127)), 0)
    run(check, what, *ties(rng, 0), 0)


@pytest.mark.parametrize("h", [1.3, 2.5, 0.1, 3.0, 1e-3, 2e-4, 12345.678, 3e7])
def test_division_by_a_spacing(check, h):
    rng = np.random.default_rng(int(h * 10))
    for lo, hi in ((-149, -110), (-60, 60), (60, 127)):
        run(check, BY_H, with_special(rng, floats(rng, lo, hi)), np.full(N, h, np.float32), 1)


@pytest.mark.parametrize("h", [0.25, 1.0, 4.0])
def test_division_by_a_power_of_two(check, h):
    rng = np.random.default_rng(2)
    run(check, BY_POW2, with_special(rng, floats(rng, -149, 127)), np.full(N, h, np.float32), 1)


def test_products_are_not_contracted(check):
    rng = np.random.default_rng(3)
    run(check, PRODUCT, floats(rng, -20, 20), floats(rng, -20, 20), 0)
    run(check, PRODUCT, with_special(rng, floats(rng, -149, 127)), with_special(rng, floats(rng, -149, 127)), 0)


def test_reciprocals(check):
    """Every divisor of the fast range."""
    res = (C.c_int * 2)()
    assert check.reciprocal_check(-10, 24, res) == 0
    assert res[0] == 0, f"{res[0]} differ, first {np.uint32(res[1]).view(np.float32)!r}"


def test_round24(check):
    """A double to float and back, below 2^126: random ones, floats, ties of floats, subnormals."""
    rng = np.random.default_rng(4)
    f = floats(rng, -149, 124).astype(np.float64)
    up = np.nextafter(f.astype(np.float32), np.float32(np.inf), dtype=np.float32).astype(np.float64)
    tie = 0.5 * (f + up)
    x = np.concatenate([f, tie, np.nextafter(tie, -np.inf), np.nextafter(tie, np.inf), f * (1 + rng.random(N) * 2.0**-20),
                        f * np.exp2(-rng.integers(0, 60, N).astype(np.float64)), [0.0, -0.0, 2.0**-150, -2.0**-150, 2.0**-1074]])
    x = np.ascontiguousarray(x)
    res = (C.c_int * 2)()
    assert check.round_check(x.ctypes.data_as(C.c_void_p), x.size, res) == 0
    assert res[0] == 0, f"{res[0]} differ, first {x[min(res[1], x.size - 1)]!r}"
