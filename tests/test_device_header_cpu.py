"""The host-callable parts of csrc/common.cuh, compiled from that header: the division by a host-known divisor,
and the plane words of the 8-wide nodes with the roundings that the traversal makes on them."""
import ctypes
import subprocess

import numpy as np
import pytest

from crt_gb300 import build

SOURCE = r"""
#include "common.cuh"
extern "C" void quotients(const uint32_t* n, size_t k, uint32_t d, uint32_t* q) {
    const FastDiv f = fast_div(d);
    for (size_t i = 0; i < k; ++i) q[i] = div_by(n[i], f);
}
extern "C" void words(const uint32_t* a, const uint32_t* b, size_t k, uint32_t* w) {
    for (size_t i = 0; i < k; ++i) w[i] = plane_word(a[i], b[i]);
}
extern "C" void planes(const double* x, size_t k, int even, int above, double* q) {
    for (size_t i = 0; i < k; ++i) q[i] = above ? plane_above(x[i], even) : plane_below(x[i], even);
}
"""


@pytest.fixture(scope="module")
def header(tmp_path_factory):
    d = tmp_path_factory.mktemp("header")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([build.NVCC, "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-I" + build.CSRC, "-I" + build.INCLUDE, str(d / "t.cu"), "-o",
                    str(d / "t.so")], check=True)
    return ctypes.CDLL(str(d / "t.so"))


def call(f, ins, *args, out):
    f(*[a.ctypes.data_as(ctypes.c_void_p) for a in ins], ctypes.c_size_t(len(ins[0])), *args,
      out.ctypes.data_as(ctypes.c_void_p))
    return out


def test_quotients_below_two_to_the_31(header):
    rng = np.random.default_rng(1)
    divisors = set(range(1, 70)) | {2 ** k + e for k in range(1, 31) for e in (-1, 0, 1)} | \
        {int(x) for x in 2.0 ** rng.uniform(0, 31, 200)}
    for d in sorted(divisors - {0}):
        k = rng.integers(0, (2 ** 31 - 1) // d + 1, 500) * d
        n = np.unique(np.concatenate([k, k + d - 1, k + 1, np.maximum(k, 1) - 1, [0, 1, 2 ** 31 - 1]]))
        n = n[n < 2 ** 31].astype(np.uint32)
        q = call(header.quotients, [n], ctypes.c_uint32(d), out=np.empty_like(n))
        np.testing.assert_array_equal(q, n // np.uint32(d))


def read(w, even):
    """The plane as the traversal reads it: 256 + quanta, exactly."""
    return (w.view(np.float32) if even else np.abs((w & 0xFFFF).astype(np.uint16).view(np.float16))).astype(np.float64)


@pytest.mark.parametrize("even", [True, False])
def test_planes_enclose_the_box_after_rounding(header, even):
    """t = fma(256 + q, s, fma(-256, s, a)) in FP32, against the distance a + x s of the box side at x quanta.
    The two roundings are at most 2^-24 (|a| + 256 |s|) and 2^-24 (|a| + 257 |s|), so with one quantum to
    spare the planes enclose the side while |a| <= 2^22 |s|."""
    rng = np.random.default_rng(5)
    n = 200_000
    x = np.concatenate([rng.uniform(2.0, 253.0, n - 1000), rng.integers(2, 254, 1000)])   # (as the collapse lays a node out)
    other = rng.integers(0, 256, n).astype(np.uint32)
    s = (2.0 ** rng.uniform(-20, 20, n) * rng.choice([-1.0, 1.0], n)).astype(np.float32).astype(np.float64)
    a = (s * 2.0 ** rng.uniform(-10, 22, n) * rng.choice([-1.0, 1.0], n)).astype(np.float32).astype(np.float64)
    c = (a - 256.0 * s).astype(np.float32).astype(np.float64)
    for above in (False, True):
        q = call(header.planes, [x], ctypes.c_int(even), ctypes.c_int(above), out=np.empty(n))
        assert q.min() >= 0 and q.max() <= 255
        q = q.astype(np.uint32)
        v = read(call(header.words, [q, other] if even else [other, q], out=np.empty_like(q)), even)
        assert np.all(np.abs(v - 256.0 - q) <= 0.75 if even else v == 256.0 + q)
        t = (v * s + c).astype(np.float32).astype(np.float64)
        side = np.sign(s) * (t - (a + x * s))   # past the side, along the axis
        assert np.all(side >= 0.0 if above else side <= 0.0)
        error = np.abs(t - (a + (v - 256.0) * s))
        assert np.all(error <= 2.0 ** -24 * (2.0 * np.abs(a) + 513.0 * np.abs(s)) * (1 + 1e-6))
