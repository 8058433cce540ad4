"""IEEE double products, quotients, comparisons and the step factor in integer
arithmetic (csrc/va_int64.cuh, csrc/va_stepfactor.cuh), built for the host and
compared bit for bit with the host's IEEE arithmetic: random operands over the
accepted range, halfway cases and their neighbours, zeros of both signs,
powers of two, and the operands that have to be refused."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("i64") / "libi64.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(ROOT, "tests", "cpp", "int64_lib.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def two(f, a, b):
    a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
    out, ok = np.empty_like(a), np.empty(len(a), np.uint8)
    f(ctypes.c_int(len(a)), ptr(a), ptr(b), ptr(out), ptr(ok))
    return out, ok.astype(bool)


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def wide(rng, n, e):
    """Random significands (half of them short, so products and quotients hit halves and exact values), exponents
    up to 2^+-e, both signs."""
    m = 1.0 + rng.random(n)
    keep = rng.integers(0, 53, n)
    short = np.ldexp(np.floor(np.ldexp(m, keep)), -keep)
    m = np.where(rng.random(n) < 0.5, short, m)
    return np.ldexp(m, rng.integers(-e, e + 1, n)) * rng.choice([-1.0, 1.0], n)


@pytest.mark.parametrize("e", [0, 3, 479])
def test_products(lib, e):
    rng = np.random.default_rng(e)
    a, b = wide(rng, 400000, e), wide(rng, 400000, e)
    # 27-bit by 27-bit significands: exact halves in the 54th bit
    a[:50000] = rng.integers(2 ** 26, 2 ** 27, 50000) * rng.choice([-1.0, 1.0], 50000)
    b[:50000] = rng.integers(2 ** 26, 2 ** 27, 50000)
    one = np.nextafter(1.0, 0.0)
    a[50000:50004], b[50000:50004] = [one, one, -one, np.nextafter(2.0, 1.0)], [one, -1.0, 1.0 / one, one]
    a[50010:50020] = [0.0, -0.0, 0.0, -0.0, 1.5, -1.5, 2.0 ** 479, 0.0, -0.0, 1.0]
    b[50010:50020] = [0.0, 0.0, -0.0, -0.0, 0.0, 0.0, -0.0, -2.0 ** 479, 2.0 ** -479, 1.0]
    out, ok = two(lib.i64_mul, a, b)
    assert ok.all()
    np.testing.assert_array_equal(bits(out), bits(a * b))


def test_products_refused(lib):
    bad = np.array([np.inf, -np.inf, np.nan, 5e-324, -2.0 ** -1050, 2.0 ** -1022, 2.0 ** -481, 2.0 ** 481, 1e300])
    for a, b in ((bad, np.full(len(bad), 1.25)), (np.full(len(bad), -3.0), bad)):
        _, ok = two(lib.i64_mul, a, b)
        assert not ok.any()


def test_quotients(lib):
    rng = np.random.default_rng(7)
    n, d = np.abs(wide(rng, 400000, 300)), np.abs(wide(rng, 400000, 300))
    n[:100000] = d[:100000] * rng.integers(1, 2 ** 20, 100000)  # near exact quotients
    q = rng.integers(2 ** 53, 2 ** 54, 100000).astype(np.float64)  # quotients near a half
    d[100000:200000] = rng.integers(1, 2 ** 20, 100000) * 2.0 + 1
    n[100000:200000] = d[100000:200000] * q
    near = 1.0 + rng.integers(-4, 5, 50000) * 2.0 ** -52
    n[200000:250000] = d[200000:250000] * near  # quotients around 1
    out, ok = two(lib.i64_div, n, d)
    assert ok.all()
    np.testing.assert_array_equal(bits(out), bits(n / d))
    bad = np.array([0.0, -1.0, np.inf, np.nan, 5e-324])
    assert not two(lib.i64_div, bad, np.ones(5))[1].any()
    assert not two(lib.i64_div, np.ones(5), bad)[1].any()
    assert not two(lib.i64_div, [1e-300], [1e300])[1].any()


def test_step_factor_decides_and_is_correctly_rounded(lib, oracle):
    """Against the oracle's binary128 power; on the controller's arguments the 2^-70 window leaves about one call in
    2^16 undecided (for K = 8, values an ulp or a few above 1 have powers within 2^-100 of a halfway point)."""
    rng = np.random.default_rng(11)
    for k in (3, 5, 6, 8):
        x = np.concatenate([10 ** rng.uniform(np.log10(5.0 ** -8), np.log10(0.5), 20000), 10 ** rng.uniform(0, 30, 10000),
                            1.0 + rng.integers(1, 100, 2000) * 2.0 ** -52, 2.0 ** rng.integers(-17, 99, 500)])
        x = x[x < 1e30]
        out, ok = np.empty_like(x), np.empty(len(x), np.uint8)
        lib.i64_pow(ctypes.c_int(k), ctypes.c_int(len(x)), ptr(x), ptr(out), ptr(ok))
        assert ok[:29000].mean() > 0.999
        want = np.array([oracle.step_pow(float(v), k, 2) for v in x])
        sel = ok.astype(bool)
        np.testing.assert_array_equal(bits(out)[sel], bits(want)[sel])


def test_comparisons(lib):
    rng = np.random.default_rng(3)
    for c in (2.220446049250313e-16, 0.5, 1.0):
        v = np.concatenate([rng.standard_normal(1000) * c, [c, np.nextafter(c, 0), np.nextafter(c, 9), -c, 0.0, -0.0,
                            np.inf, -np.inf, np.nan, -np.nan, 5e-324]])
        out = np.empty(len(v), np.uint8)
        lib.i64_cmp(ctypes.c_int(len(v)), ptr(v), ctypes.c_double(c), ptr(out))
        np.testing.assert_array_equal((out & 1) != 0, v > c)
        np.testing.assert_array_equal((out & 2) != 0, v <= c)
        np.testing.assert_array_equal((out & 4) != 0, np.isnan(v))
        np.testing.assert_array_equal((out & 8) != 0, np.isfinite(v))
