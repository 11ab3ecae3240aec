"""The integer FP64 product and quotient of the FP64 velocity sums (csrc/fp64_int.cuh), compiled for
the host, against the host's own IEEE arithmetic: bit for bit, on random mantissas, on mantissas
with long runs of zeros and ones (ties, carries to the next power) and on neighbours of exact
quotients."""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import PKG

SRC = """
#include "fp64_int.cuh"
extern "C" void both(long n, const double* a, const double* b, double* p, double* f, double* q) {
  for (long i = 0; i < n; ++i) {
    const lpm::F64Parts pa = lpm::f64_parts(a[i]);
    const lpm::F64Factor fb = lpm::f64_factor(lpm::f64_parts(b[i]));
    p[i] = lpm::mul_rn_int<true>(pa, fb);
    f[i] = lpm::f64_short(a[i]) || lpm::f64_short(b[i]) ? a[i] * b[i] : lpm::mul_rn_int<false>(pa, fb);
    const unsigned long long w = lpm::f64_bits(b[i]);
    q[i] = lpm::div_rn_int(pa, lpm::F64Words{static_cast<uint32_t>(w), static_cast<uint32_t>(w >> 32)});
  }
}
"""


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64_int")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", "-I",
                    str(PKG / "csrc"), str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    fn = ctypes.CDLL(str(d / "t.so")).both

    def call(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        out = [np.empty_like(a) for _ in range(3)]
        ptr = [v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, *out)]
        fn(ctypes.c_long(a.size), *ptr)
        return out
    return call


def _doubles(rng, n, kind):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    s = rng.integers(0, 52, n, dtype=np.uint64)
    if kind == "zeros":
        m = (m >> s) << s
    elif kind == "ones":
        m |= (np.uint64(1) << s) - np.uint64(1)
    elif kind == "edge":
        m = np.where(rng.random(n) < 0.5, np.uint64((1 << 52) - 1) - (m % np.uint64(4)), m % np.uint64(4))
    e = rng.integers(1023 - 100, 1023 + 100, n).astype(np.uint64)
    sign = rng.integers(0, 2, n).astype(np.uint64)
    return ((sign << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


@pytest.mark.parametrize("ka", ["any", "zeros", "ones", "edge"])
@pytest.mark.parametrize("kb", ["any", "zeros", "ones", "edge"])
def test_product_and_quotient_are_the_ieee_ones(both, ka, kb):
    rng = np.random.default_rng([len(ka), len(kb), ord(ka[0]), ord(kb[0])])
    a, b = _doubles(rng, 300000, ka), _doubles(rng, 300000, kb)
    p, f, q = both(a, b)
    assert np.array_equal(p, a * b)
    assert np.array_equal(f, a * b)
    assert np.array_equal(q, a / b)


def test_quotients_next_to_a_double(both):
    """Numerators one ulp around an exact product: quotients just above and below a double."""
    rng = np.random.default_rng(7)
    b, c = _doubles(rng, 300000, "any"), _doubles(rng, 300000, "zeros")
    for a in (b * c, np.nextafter(b * c, np.inf), np.nextafter(b * c, -np.inf)):
        assert np.array_equal(both(a, b)[2], a / b)


def test_products_next_to_the_next_power(both):
    """a b just below 2: the product rounds up to the power."""
    rng = np.random.default_rng(8)
    a = 1.0 + rng.random(300000)
    b = np.nextafter(2.0 / a, 0.0)
    for v in (b, 2.0 / a, np.nextafter(2.0 / a, 4.0)):
        p, f, _ = both(a, v)
        assert np.array_equal(p, a * v) and np.array_equal(f, a * v)
