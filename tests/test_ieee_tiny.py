"""Quotients of dividends below 2^-300 in swehr_ieee.h: sw_quot down to 2^-860
over a depth or a constant (and that quotient over a constant again), and
sw_quot_tiny down to the smallest subnormal, where a result has few bits, lies on
a midpoint of two subnormals or next to one.  On the CPU with any estimate within
2^-18, on the GPU with the hardware's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_ieee_quotients import PKG, _ptr, random_pairs

CHECK = r"""
#include <stdint.h>
#include "swehr_ieee.h"
static uint64_t next(uint64_t *s) { *s ^= *s << 13; *s ^= *s >> 7; *s ^= *s << 17; return *s; }
static double rough(double v, uint64_t *s)
{
    const double d = ((double)(next(s) >> 11) * 0x1p-52 - 1.0) * 0x1p-18;
    return sw_from_bits(sw_bits(v * (1 + d)) & (long long)0xffffffff00000000ull);
}
int64_t check(int tiny, const double *a, const double *b, int64_t n, int rounds, uint64_t seed)
{
    int64_t bad = 0;
    for (int64_t k = 0; k < n; k++)
        for (int r = 0; r < rounds; r++) {
            const double y = sw_rcp_refine(b[k], rough(1.0 / b[k], &seed));
            bad += sw_bits(tiny ? sw_quot_tiny(a[k], b[k], y) : sw_quot(a[k], b[k], y)) != sw_bits(a[k] / b[k]);
        }
    return bad;
}
"""


def low_pairs(n, seed):
    """dividends in [2^-860, 2^-300), divisors in [2^-200, 2^52)"""
    rng = np.random.default_rng(seed)
    a = rng.uniform(1, 2, n) * np.exp2(rng.integers(-860, -300, n)) * rng.choice([-1.0, 1.0], n)
    b = rng.uniform(1, 2, n) * np.exp2(rng.integers(-200, 52, n))
    a[::5] = np.copysign(2.0 ** -860, a[::5])
    b[::7] = 2.0 ** 52 * (1 - 2.0 ** -53)
    b[1::7] = 2.0 ** -200
    return a, b


def subnormal_pairs(n, seed):
    rng = np.random.default_rng(seed)
    tiny = 2.0 ** -1074
    few = rng.integers(0, 40, n) * tiny                         # a few units
    a = np.concatenate([few, rng.integers(1, 2 ** 52, n) * tiny, rng.uniform(1, 2, n) * np.exp2(rng.integers(-1074, -850, n))])
    b = rng.uniform(1, 2, a.size) * np.exp2(rng.integers(-40, 52, a.size))
    b[:n:2] = rng.integers(1, 64, b[:n:2].size) / 16.0           # exact ties among them
    a *= rng.choice([-1.0, 1.0], a.size)
    # quotients k + 1/2 units, exactly and one unit of the dividend beside it
    k = rng.integers(0, 2 ** 20, n).astype(np.float64)
    half = rng.integers(1, 1 << 20, n).astype(np.float64)        # b = 2 half: a = (2k + 1) half units
    ta = (2 * k + 1) * half
    ties_a = np.concatenate([ta, ta + 1, ta - 1]) * tiny
    ties_b = np.tile(2 * half, 3)
    # the same with dividends of 53 bits: a 2^p = b (2q + 1) + c, p bits short of the last place
    A, B = [], []
    for Bi in (int(v) | 1 for v in rng.integers(1 << 52, 1 << 53, 400)):
        for p in range(1, 52, 3):
            inv = pow(2, -p, Bi)
            for c in (-3, -1, 1, 3):
                A0 = c * inv % Bi
                if (1 << 52) <= A0 and ((A0 << p) - c) // Bi % 2 == 1:
                    A.append(float(A0) * 2.0 ** -1074)           # [2^-1022, 2^-1021)
                    B.append(float(Bi) * 2.0 ** (-p + 1))
    A, B = np.array(A), np.array(B)
    for shift in (-1, 0, 1, 2):
        ok = (B * 2.0 ** shift < 2.0 ** 52) & (B * 2.0 ** shift >= 2.0 ** -200)
        ties_a, ties_b = np.concatenate([ties_a, A[ok]]), np.concatenate([ties_b, B[ok] * 2.0 ** shift])
    return np.concatenate([a, ties_a]), np.concatenate([b, ties_b])


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiny")
    src, so = str(d / "check.c"), str(d / "check.so")
    with open(src, "w") as f:
        f.write(CHECK)
    subprocess.check_call(["gcc", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unused-variable",
                           "-I", os.path.join(PKG, "csrc"), src, "-o", so, "-lm"])
    L = C.CDLL(so)
    pd = C.POINTER(C.c_double)
    L.check.restype = C.c_int64
    L.check.argtypes = [C.c_int, pd, pd, C.c_int64, C.c_int, C.c_uint64]
    return L


def test_low_dividends_on_the_host(host):
    a, b = low_pairs(400000, 31)
    assert host.check(0, _ptr(a), _ptr(b), a.size, 2, 41) == 0
    q, c = a / b, np.full_like(a, 2600.0)                         # TOTSED: U_k / h / rhos
    for rhos in (2600.0, 2.0 ** 50 * (1 - 2.0 ** -53), 2.0 ** -100):
        c[:] = rhos
        assert host.check(0, _ptr(q), _ptr(c), q.size, 1, 42) == 0


def test_tiny_dividends_on_the_host(host):
    a, b = subnormal_pairs(200000, 32)
    q = np.abs(a / b)
    assert (q < 2.0 ** -1022).sum() > 400000 and (q == 0).sum() > 1000
    assert host.check(1, _ptr(a), _ptr(b), a.size, 2, 43) == 0
    a, b = low_pairs(100000, 33)
    assert host.check(1, _ptr(a), _ptr(b), a.size, 2, 44) == 0
    a, b = random_pairs(200000, 34, span=190)
    b = np.where(b < 2.0 ** 52, b, 1.5)
    assert host.check(1, _ptr(a), _ptr(b), a.size, 1, 45) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("op", ["low", "tiny", "exp"])
def test_device_results_equal_the_operators(op):
    L = C.CDLL(os.path.join(PKG, "libswehr_probe.so"))
    pd = C.POINTER(C.c_double)
    L.swehr_probe_ieee.restype = C.c_int
    L.swehr_probe_ieee.argtypes = [C.c_int, pd, pd, C.c_int64, pd, pd, pd]
    if op == "exp":                                               # below -746: zero
        a = np.concatenate([-746.0 - 10.0 ** np.random.default_rng(37).uniform(-2.9, 9, 400000), [-746.0011, -1e200]])
        b = np.ones_like(a)
    else:
        a, b = low_pairs(2000000, 35) if op == "low" else subnormal_pairs(400000, 36)
    fast, plain, refused = np.empty_like(a), np.empty_like(a), np.empty_like(a)
    assert L.swehr_probe_ieee({"low": 5, "tiny": 6, "exp": 7}[op], _ptr(a), _ptr(b), a.size, _ptr(fast), _ptr(plain), _ptr(refused)) == 0
    assert not refused.any()
    want = np.zeros_like(a) if op == "exp" else a / b
    assert np.array_equal(plain.view(np.int64), want.view(np.int64))
    assert np.array_equal(fast.view(np.int64), plain.view(np.int64))
