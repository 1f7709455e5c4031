"""The branch-free quotients and square roots of swehr_ieee.h give the IEEE
results: on the CPU against the host's operators (any estimate within 2^-18),
on the GPU, with the hardware's estimates, against the compiler's operators.

Random operands say little about a rounding that only fails near a midpoint of
two doubles, so the operands whose quotients and roots lie nearest to one are
constructed: a 2^53 = b (2q+1) + c and a 2^54 = b (2q+1) + c for small c, and
k^2 = -c modulo 2^54 and 2^55, k odd.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "swehr_b200")

CHECK = r"""
#include <stdint.h>
#include "swehr_ieee.h"
static uint64_t next(uint64_t *s) { *s ^= *s << 13; *s ^= *s >> 7; *s ^= *s << 17; return *s; }
/* an estimate of v, relatively off by up to 2^-18, low word zero as the hardware's */
static double rough(double v, uint64_t *s)
{
    const double d = ((double)(next(s) >> 11) * 0x1p-52 - 1.0) * 0x1p-18;
    return sw_from_bits(sw_bits(v * (1 + d)) & (long long)0xffffffff00000000ull);
}
static int same(double x, double y) { return sw_bits(x) == sw_bits(y) || (x != x && y != y); }
int64_t check_div(const double *a, const double *b, int64_t n, int rounds, uint64_t seed)
{
    int64_t bad = 0;
    for (int64_t k = 0; k < n; k++)
        for (int r = 0; r < rounds; r++)
            bad += !same(sw_quot(a[k], b[k], sw_rcp_refine(b[k], rough(1.0 / b[k], &seed))), a[k] / b[k]);
    return bad;
}
int64_t check_sqrt(const double *x, int64_t n, int rounds, uint64_t seed)
{
    int64_t bad = 0;
    for (int64_t k = 0; k < n; k++)
        for (int r = 0; r < rounds; r++)
            bad += !same(sw_sqrt_refine(x[k], rough(1.0 / sqrt(x[k]), &seed)), sqrt(x[k]));
    return bad;
}
"""


def random_pairs(n, seed, span=299):
    rng = np.random.default_rng(seed)
    a = rng.uniform(1, 2, n) * np.exp2(rng.integers(-span, span, n)) * rng.choice([-1.0, 1.0], n)
    b = rng.uniform(1, 2, n) * np.exp2(rng.integers(-span, span, n))
    a[:: 97] = 0.0
    a[1:: 97] = -0.0
    a[2:: 97] = b[2:: 97]
    return a, b


def hard_pairs(count, seed):
    """a/b within a few units of the smallest possible distance from a midpoint."""
    rng = np.random.default_rng(seed)
    top = 1 << 53
    divisors = [int(v) | 1 for v in rng.integers(1 << 52, top, count)]
    divisors += [top - k for k in range(1, 200, 2)] + [(1 << 52) + k for k in range(1, 200, 2)]
    a, b = [], []
    for B in divisors:
        for shift in (53, 54):
            inv = pow(2, -shift, B)
            for c in range(-9, 10, 2):
                A0 = c * inv % B
                for A in (A0, A0 + B):
                    if (1 << 52) <= A < top and ((A << shift) - c) // B % 2 == 1:
                        a.append(float(A))
                        b.append(float(B))
    return np.array(a), np.array(b)


def _root(c, n):
    """r with r^2 = c modulo 2^n (c = 1 modulo 8)."""
    r = 1
    for k in range(3, n):
        if (r * r - c) % (1 << (k + 1)):
            r += 1 << (k - 1)
    assert (r * r - c) % (1 << n) == 0
    return r


def hard_roots(limit=2000):
    """x whose root k 2^-53 (k odd) differs from a midpoint by |c| < limit units of the last place of k^2."""
    xs = []
    for c in range(-limit, limit):
        if (-c) % 8 != 1:
            continue
        for n, lo, hi in ((54, 1 << 53, int(2 ** 53.5)), (55, int(2 ** 53.5), 1 << 54)):
            r = _root(-c % (1 << n), n)
            for k in {r, -r, r + (1 << (n - 1)), -r + (1 << (n - 1))}:
                k %= 1 << n
                if lo <= k < hi and ((k * k + c) >> n) < (1 << 53):
                    xs.append(float((k * k + c) >> n) * (1.0 if n == 54 else 2.0))
    return np.array(xs)


def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("ieee")
    src, so = str(d / "check.c"), str(d / "check.so")
    with open(src, "w") as f:
        f.write(CHECK)
    subprocess.check_call(["gcc", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unused-variable",
                           "-I", os.path.join(PKG, "csrc"), src, "-o", so, "-lm"])
    L = C.CDLL(so)
    pd = C.POINTER(C.c_double)
    L.check_div.restype = L.check_sqrt.restype = C.c_int64
    L.check_div.argtypes = [pd, pd, C.c_int64, C.c_int, C.c_uint64]
    L.check_sqrt.argtypes = [pd, C.c_int64, C.c_int, C.c_uint64]
    return L


def test_quotients_on_the_host(host):
    a, b = random_pairs(400000, 1)
    assert host.check_div(_ptr(a), _ptr(b), a.size, 2, 11) == 0
    a, b = hard_pairs(4000, 2)
    assert a.size > 10000
    assert host.check_div(_ptr(a), _ptr(b), a.size, 8, 12) == 0
    scaled = b * 2.0 ** -300
    assert host.check_div(_ptr(a), _ptr(scaled), a.size, 2, 13) == 0


def test_roots_on_the_host(host):
    a, b = random_pairs(400000, 3)
    assert host.check_sqrt(_ptr(b), b.size, 2, 21) == 0
    x = hard_roots()
    assert x.size > 500
    for scale in (1.0, 2.0 ** -40, 2.0 ** 202):
        y = x * scale
        assert host.check_sqrt(_ptr(y), y.size, 64, 22) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["div", "sqrt", "exp", "pow", "cos_atan"])
def test_device_results_equal_the_plain_operators(op):
    L = C.CDLL(os.path.join(PKG, "libswehr_probe.so"))
    pd = C.POINTER(C.c_double)
    L.swehr_probe_ieee.restype = C.c_int
    L.swehr_probe_ieee.argtypes = [C.c_int, pd, pd, C.c_int64, pd, pd, pd]
    rng = np.random.default_rng(5)
    if op == "div":
        sets = [random_pairs(2000000, 4), hard_pairs(8000, 6)]
    elif op == "sqrt":
        x = random_pairs(2000000, 7)[1]
        x[::101] = 0.0
        x[1::101] = -0.0
        h = hard_roots()
        sets = [(x, x), (h, h), (h * 2.0 ** -60, h)]
    elif op == "exp":
        x = np.concatenate([rng.uniform(-700, 700, 500000), rng.uniform(-50, 0, 500000),
                            10 ** rng.uniform(-300, 0, 200000), [0.0, -0.0]])
        sets = [(x, x)]
    elif op == "pow":
        x = np.concatenate([10 ** rng.uniform(-8, 3, 500000), rng.uniform(0.9, 1.1, 200000), [1.0, 2.0, 0.5]])
        sets = [(x, np.full_like(x, y)) for y in (3.333, 2.333, -0.33, 0.6, -2.5, 0.0)]
    else:
        x = np.concatenate([rng.uniform(-3, 3, 500000), 10 ** rng.uniform(-200, 100, 200000), [0.0]])
        sets = [(x, x)]
    for a, b in sets:
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        fast, plain, refused = np.empty_like(a), np.empty_like(a), np.empty_like(a)
        assert L.swehr_probe_ieee(["div", "sqrt", "exp", "pow", "cos_atan"].index(op), _ptr(a), _ptr(b), a.size,
                                  _ptr(fast), _ptr(plain), _ptr(refused)) == 0
        assert not refused.any()
        bad = fast.view(np.int64) != plain.view(np.int64)
        assert not bad.any(), (op, int(bad.sum()), a[bad][:3], b[bad][:3], fast[bad][:3], plain[bad][:3])
        if op == "div":
            assert np.array_equal(plain, a / b)
        if op == "sqrt":
            assert np.array_equal(plain, np.sqrt(a))
