"""divisor.h (the diffusion adjoint's quotients) against the division it
stands for, bit for bit, compiled for the host."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = """
#include "divisor.h"
extern "C" void divide(const float* x, const float* z, float* q, long n) {
    for (long i = 0; i < n; ++i) {
        bool divide = false;
        q[i] = cg::Divisor(z[i]).quotient(x[i], &divide);
        if (divide) q[i] = x[i] / z[i];
    }
}
"""


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    d = tmp_path_factory.mktemp("divisor")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "cella_nova_gb300", "csrc"), "shim.cpp", "-o", "shim.so"],
                   cwd=d, check=True)
    lib = ctypes.CDLL(str(d / "shim.so"))

    def call(x, z):
        x, z = (np.ascontiguousarray(a, np.float32) for a in np.broadcast_arrays(x, z))
        q = np.empty_like(x)
        p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))
        lib.divide(p(x), p(z), p(q), ctypes.c_long(x.size))
        return q
    return call


def same_bits(divide, x, z):
    x, z = np.broadcast_arrays(np.asarray(x, np.float32), np.asarray(z, np.float32))
    got = divide(x, z)
    with np.errstate(all="ignore"):
        want = x / z
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])


def around(*values):
    v = np.array(values, np.float32)
    with np.errstate(all="ignore"):
        v = np.concatenate([v, np.nextafter(v, np.float32(np.inf)),
                            np.nextafter(v, np.float32(-np.inf))])
    return np.concatenate([v, -v])


def test_ends_of_every_range(divide):
    x = around(0, 2.0 ** -149, 2.0 ** -127, 2.0 ** -126, 2.0 ** -101, 2.0 ** -100, 1 / 3, 1, 7,
               2.0 ** 100, 2.0 ** 101, 2.0 ** 127, np.inf, np.nan, np.finfo(np.float32).max)
    z = around(0, 2.0 ** -149, 2.0 ** -126, 2.0 ** -25, 2.0 ** -24, 0.3, 1, 9, 2.0 ** 24,
               2.0 ** 25, 2.0 ** 127, np.inf, np.nan)
    same_bits(divide, x[:, None], z[None, :])


@pytest.mark.parametrize("seed", [1, 2])
def test_any_bits(divide, seed):
    x, z = np.random.default_rng(seed).integers(0, 1 << 32, (2, 1 << 20), dtype=np.uint32)
    same_bits(divide, x.view(np.float32), z.view(np.float32))
    # divisors as the diffusion has them
    z = np.exp(np.random.default_rng(seed).uniform(-8, 8, x.size)).astype(np.float32)
    same_bits(divide, x.view(np.float32), z)


@pytest.mark.parametrize("c", [-3, -1, 1, 3])
def test_quotients_next_to_a_rounding_boundary(divide, c):
    """Numerators with 2^(s+1) x = z (2 Q + 1) + c for a 24-bit Q: the quotient
    is c / (2 z) of its last place away from the middle of two numbers."""
    z = np.random.default_rng(9).integers(1 << 22, 1 << 23, 1 << 18, dtype=np.uint64) * 2 + 1
    inv = np.ones_like(z)
    for _ in range(6):   # z^-1 modulo 2^64
        inv *= 2 - z * inv
    found = 0
    for s in (23, 24):
        mid = np.uint64(-c % (1 << 64)) * inv & np.uint64((1 << (s + 1)) - 1)
        x = (z * mid + np.uint64(c % (1 << 64))) >> np.uint64(s + 1)
        ok = (mid >= 1 << 24) & (mid < 1 << 25) & (x > 0) & (x < 1 << 24)
        found += int(ok.sum())
        same_bits(divide, x[ok].astype(np.float32), z[ok].astype(np.float32))
    assert found > 1 << 16
