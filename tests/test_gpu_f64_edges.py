"""FP64 building blocks at the ends of their ranges (NaN, infinities, numbers
whose products overflow, empty and reversed tables) give the bits of the plain
operations they stand for, and scenes that reach them give the frames they
gave before the blocks were written. Exact but where a bound is given."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "device_f64_edges.cu")
OUT = os.path.join(ROOT, "_build", "test", "libf64edges.so")
NAN, INF = np.nan, np.inf


@pytest.fixture(scope="module")
def edges(need_gpu):
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-shared", "-cudart", "static", "-Xcompiler", "-fPIC", "-ccbin", "/usr/bin/g++", "-o", OUT, SRC],
                   check=True)
    lib = C.CDLL(OUT)

    def run(kind, rows):
        rows = np.ascontiguousarray(rows, dtype=np.float64)
        fast, plain = np.empty((len(rows), 2)), np.empty((len(rows), 2))
        p = [a.ctypes.data_as(C.c_void_p) for a in (rows, fast, plain)]
        assert lib.f64_edges(kind, p[0], len(rows), p[1], p[2]) == 0
        return rows, fast, plain

    return run


def assert_same(result):
    """Equal bits, any NaN like any other."""
    rows, fast, plain = result
    same = (fast.view(np.uint64) == plain.view(np.uint64)) | (np.isnan(fast) & np.isnan(plain))
    bad = np.nonzero(~same.all(axis=1))[0]
    assert len(bad) == 0, (len(bad), rows[bad[:4]], fast[bad[:4]], plain[bad[:4]])


def test_reciprocal_of_nan_and_infinity(edges):
    odd = [NAN, -NAN, INF, -INF, 1.0, -3.0, 2.0 ** 1022, 2.0 ** 1023]
    x = [v for v in odd if not 2.0 ** 1022 <= abs(v) < INF] + [2.0 ** 1021]  # results of normal range, or 0
    assert_same(edges(0, [(a, b) for a in odd + [0.0] for b in x]))


def test_right_hand_side_of_nan_is_nan(edges):
    assert_same(edges(4, [(r, th, pr, pth) for r, th in ((NAN, 1.2), (6.0, NAN), (NAN, NAN), (-NAN, 0.0))
                          for pr in (0.0, -0.7, INF) for pth in (0.0, 1.3, -INF)]))


@pytest.mark.parametrize("top", [1e3, 1e150, 1e160, 1e300])
def test_largest_quotient(edges, top):
    rng = np.random.default_rng(11)
    n = 20000
    span = np.log10(top)
    rows = np.concatenate([10.0 ** rng.uniform(-30, span, (n, 5)), 10.0 ** rng.uniform(-12, span, (n, 5))], axis=1)
    odd = rng.random((n, 10)) < 0.05
    rows[odd] = rng.choice([0.0, NAN, INF, -INF, 1e-9, top], int(odd.sum()))
    rows *= np.where(rng.random((n, 10)) < 0.5, -1.0, 1.0)
    assert_same(edges(1, rows))


def test_table_cell_of_infinite_coordinates(edges):
    rng = np.random.default_rng(12)
    rows = [(lv, 13.0, 19.3, 60) for lv in (INF, -INF, NAN, 13.0, 19.3, np.nextafter(19.3, 20), 12.9, -323.0, 308.2)]
    rows += [(lv, -18.0, -6.0, 100) for lv in (INF, -INF, NAN, 0.0, -0.0, -18.0, -6.0, -320.0)]
    rows += [(lv, 13.0, 19.3, 60) for lv in rng.uniform(12.0, 21.0, 20000)]
    assert_same(edges(2, rows))


def test_radial_table_at_and_beyond_its_ends(edges):
    rng = np.random.default_rng(13)
    rows = []
    for lo, hi in ((1.4459, 30.0), (2.01, 2.01), (2.01, 1.5), (2.01, np.nextafter(2.01, 3))):
        r = [lo, hi, np.nextafter(lo, 0), np.nextafter(lo, 9), np.nextafter(hi, 0), np.nextafter(hi, 99), 0.0, 1e3,
             INF, NAN] + list(rng.uniform(0.9 * min(lo, hi), 1.2 * max(lo, hi), 2000))
        rows += [(v, lo, hi) for v in r]
    assert_same(edges(3, rows))


def spectral(grrt, bins, **kw):
    """A small cube at the given bins, tables laid out for ordinary ones."""
    R = grrt.Renderer(grrt.config_params(3, width=32, height=24, **kw), freqs=grrt.log_bins(n=4))
    R.freqs = np.array(bins, dtype=np.float64)
    grrt.lib().grrt_set_frequency_bins(R.ctx, R.freqs.ctypes.data_as(C.POINTER(C.c_double)), len(bins))
    return R.render_spectral(), R.stats()


@pytest.mark.parametrize("odd,like", [(0.0, 1e-3), (INF, 1e300)])
def test_a_bin_at_the_end_of_the_range_leaves_the_others(grrt, need_gpu, odd, like):
    """The opacity of a frequency below (above) the table is the table's end, so
    a bin at 0 (infinity) steers the march as any other frequency out there."""
    f = grrt.log_bins(n=4)
    a, sa = spectral(grrt, [f[0], f[1], odd, f[2]])  # the third of four is the one that sets the step length
    b, sb = spectral(grrt, [f[0], f[1], like, f[2]])
    others = [0, 1, 3]
    assert (b[..., others] > 0).any()
    np.testing.assert_array_equal(a[..., others], b[..., others])
    for key in ("attempts", "march_steps", "physics_steps", "bin_updates"):
        assert sa[key] == sb[key], key


def test_an_infinite_noise_scale_is_uniform_matter(grrt, need_gpu):
    """All coordinates of the noise are 0, and the noise is continuous there: at
    1e30 they are at most 1e-28, which moves it by less than 1e-25."""
    f = grrt.log_bins(n=4)
    a, sa = spectral(grrt, f, disk_noise_scale=INF)
    b, sb = spectral(grrt, f, disk_noise_scale=1e30)
    assert sa["physics_steps"] > 0
    assert (b > 0).any()
    np.testing.assert_allclose(a, b, rtol=1e-9, atol=0.0)
