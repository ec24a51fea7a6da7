"""The FP64 right-hand side's branch-free building blocks give the bits of the
operations they stand for: the sine and cosine of the reference's polynomial
with the pole clamp, the IEEE reciprocal and quotient, and the step
controller's decision from the unformed error quotient. The expected values
are the plain operations on the same device, so every comparison is exact."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "device_f64_bits.cu")
OUT = os.path.join(ROOT, "_build", "test", "libf64bits.so")


@pytest.fixture(scope="module")
def bits(need_gpu):
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-shared", "-cudart", "static", "-Xcompiler", "-fPIC", "-ccbin", "/usr/bin/g++", "-o", OUT, SRC],
                   check=True)
    return C.CDLL(OUT)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _same(fast, plain):
    """Equal bits, any NaN like any other."""
    return (fast.view(np.uint64) == plain.view(np.uint64)) | (np.isnan(fast) & np.isnan(plain))


def _angles(kind):
    rng = np.random.default_rng(5)
    if kind == "random":
        return rng.uniform(-40.0, 40.0, 200000)
    if kind == "octants":  # where the octant changes, a few ulp to both sides
        x = np.arange(-64, 65) * (np.pi / 4)
        return np.concatenate([x] + [np.nextafter(x, s * np.inf) for s in (-1, 1)])
    if kind == "poles":
        near = np.concatenate([10.0 ** rng.uniform(-20, -2, 2000), [0.0, 1e-10, np.nextafter(1e-10, 0)]])
        return np.concatenate([base + sign * near for base in (0.0, np.pi, 2 * np.pi) for sign in (1, -1)]) + 0.0
    # past the range of a 32-bit octant: both give the same leftovers
    return np.concatenate([10.0 ** rng.uniform(6, 21, 5000), [1686629713.0, 1686629714.0, 4.0e9]])


@pytest.mark.parametrize("kind", ["random", "octants", "poles", "huge"])
def test_sincos_bits(bits, kind):
    x = np.ascontiguousarray(_angles(kind))
    fast, plain = np.empty(2 * len(x)), np.empty(2 * len(x))
    assert bits.f64_sincos(_ptr(x), len(x), _ptr(fast), _ptr(plain)) == 0
    assert np.all(_same(fast, plain))


@pytest.mark.parametrize("span", [1.0, 60.0, 300.0])
def test_reciprocal_and_quotient_bits(bits, span):
    rng = np.random.default_rng(6)
    n = 300000
    a, b = (np.where(rng.random(n) < 0.5, -1.0, 1.0) * rng.uniform(1, 10, n) * 10.0 ** rng.uniform(-span, span, n)
            for _ in range(2))
    ones = np.array([1.0, 2.0, np.nextafter(2.0, 0), np.nextafter(1.0, 2), np.inf, -np.inf])
    b = np.concatenate([b, ones, np.nextafter(2.0 ** np.arange(-200.0, 200.0), 0)])
    a = np.concatenate([a, np.ones(len(b) - len(a))])
    fast, plain = np.empty(2 * len(b)), np.empty(2 * len(b))
    assert bits.f64_divide(_ptr(a), _ptr(b), len(b), _ptr(fast), _ptr(plain)) == 0
    assert np.all(_same(fast, plain))


@pytest.mark.parametrize("tol", [1e-4, 1e-8, 1e-12, 1e-27])
def test_step_decision_bits(bits, tol):
    rng = np.random.default_rng(7)
    n = 200000
    den = 10.0 ** rng.uniform(-10, 4, n)
    err = tol * 10.0 ** rng.uniform(-6, 6, n)
    edge = rng.random(n) < 0.2  # err at tol, to a few ulp
    err[edge] = tol * (1.0 + rng.integers(-40, 41, int(edge.sum())) * 2.0 ** -52)
    num = err * den
    odd = [0.0, 1e-320, 1e300, np.inf, np.nan]
    num = np.concatenate([num, odd, odd])
    den = np.concatenate([den, np.ones(5), np.full(5, np.inf)])
    m = len(num)
    dl = 10.0 ** rng.uniform(-7, 3, m)
    retry = rng.choice([0, 1, 19, 20], m).astype(np.int32)
    r = np.where(rng.random(m) < 0.1, -1.0, 1.0) * 10.0 ** rng.uniform(-1, 3, m)
    fast, plain = np.empty(2 * m), np.empty(2 * m)
    assert bits.f64_control(_ptr(num), _ptr(den), _ptr(dl), _ptr(retry), _ptr(r), C.c_double(tol), m, _ptr(fast),
                            _ptr(plain)) == 0
    assert np.all(_same(fast, plain))
