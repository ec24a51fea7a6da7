"""The device's right-hand sides, the DP45 attempt in each of its forms and the
RK4 step give the bits of the generic bodies that they stand for, on states
such as rays pass through. Exact comparisons."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NATIVE = os.path.join(ROOT, "tests", "native")
OUT = os.path.join(ROOT, "_build", "test", "libattemptbits.so")
RHS_F32, RHS_F64, ATTEMPT, RK4 = range(4)


@pytest.fixture(scope="module")
def bits(need_gpu):
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-shared", "-cudart", "static", "-Xcompiler", "-fPIC", "-ccbin", "/usr/bin/g++", "-o", OUT,
                    os.path.join(NATIVE, "device_attempt_bits.cu"), os.path.join(NATIVE, "device_attempt_generic.cu")],
                   check=True)
    return C.CDLL(OUT)


def states(n, seed, wild):
    """M, a, p_t, p_phi, r, theta, phi, p_r, p_theta, step: photons of about unit
    energy between the horizon and the escape radius. Ordinary ones keep off the
    axis and step by a part of the distance to the horizon; wild ones take any
    step from anywhere, momenta that no light cone has, so that stages overflow."""
    rng = np.random.default_rng(seed)
    M = np.where(rng.random(n) < 0.5, 1.0, rng.uniform(0.5, 2.0, n))
    a = M * np.where(rng.random(n) < 0.2, 0.0, rng.uniform(0.0, 0.998, n))
    rh = M + np.sqrt(M * M - a * a)
    r = rh + 0.011 * M + M * 10.0 ** rng.uniform(-2, 3, n)
    th = rng.uniform(0.05, np.pi - 0.05, n) + np.where(rng.random(n) < 0.2, 2 * np.pi * rng.integers(-2, 3, n), 0.0)
    pr, pth, pph = rng.normal(0.0, 1.0, n), rng.normal(0.0, 5.0, n), rng.normal(0.0, 5.0, n)
    h = (r - rh) * 10.0 ** rng.uniform(-5, -1.5, n)
    if wild:
        th = np.where(rng.random(n) < 0.3, 10.0 ** rng.uniform(-6, -1, n), th)
        pr *= np.where(rng.random(n) < 0.1, 30.0, 1.0)
        h = 10.0 ** rng.uniform(-4, 2, n)
    return np.ascontiguousarray(np.stack([M, a, -rng.uniform(0.7, 1.2, n), pph, r, th, rng.uniform(0.0, 50.0, n), pr,
                                          pth, h], axis=1))


FORMS = [(RHS_F32, 0, 0), (RHS_F64, 0, 0), (ATTEMPT, 0, 0), (ATTEMPT, 1, 0), (ATTEMPT, 1, 1), (RK4, 0, 0),
         (RK4, 1, 0)]


@pytest.mark.parametrize("wild", [False, True])
@pytest.mark.parametrize("kind,shared,rolled", FORMS)
def test_bits_of_the_generic_form(bits, kind, shared, rolled, wild):
    n = 1 << 17
    rows = states(n, 21, wild)
    fast, plain = np.empty((n, 11)), np.empty((n, 11))
    p = [x.ctypes.data_as(C.c_void_p) for x in (rows, fast, plain)]
    assert bits.attempt_bits(kind, shared, rolled, p[0], n, p[1], p[2]) == 0
    same = (fast.view(np.uint64) == plain.view(np.uint64)) | (np.isnan(fast) & np.isnan(plain))
    # a reciprocal below the normal range counts as 0 in the right-hand side:
    # states whose derivatives or ends lie past 1e30 are left out
    with np.errstate(invalid="ignore"):
        judged = ~(np.abs(np.where(np.isnan(plain), 0.0, plain)) > 1e30).any(axis=1)
    assert judged.mean() > (0.9 if wild else 0.9999)
    if wild and kind == ATTEMPT:
        assert np.isnan(plain[judged]).any(axis=1).sum() > 100  # stages did overflow
    bad = np.nonzero(~same.all(axis=1) & judged)[0]
    assert len(bad) == 0, (len(bad), rows[bad[:2]], fast[bad[:2]], plain[bad[:2]])
