"""An FP64 thin-disk batch that nobody gave a schedule gives the frames and the
counters of one that was told to go pixel by pixel, at sizes around a warp, and
reports the same default schedule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,spp", [([(1, 1)], 1), ([(31, 1), (1, 33)], 4), ([(17, 9), (40, 30), (5, 3)], 1),
                                       ([(64, 48)] * 3, 9)])
def test_default_schedule_matches_pixels(need_gpu, grrt, sizes, spp):
    params = [grrt.config_params(2, width=w, height=h, spp=spp, spin=0.3 + 0.2 * k) for k, (w, h) in enumerate(sizes)]
    B, P = grrt.Batch(params), grrt.Batch(params)
    assert B.schedule() == P.schedule() == (256, B.ORDER_ROUND_ROBIN, 0)
    P.set_schedule(*P.schedule())
    for _ in range(2):  # the first render and a replay
        got, want = B.render(), P.render()
        for k, (g, w) in enumerate(zip(got, want)):
            np.testing.assert_array_equal(g, w, err_msg=f"camera {k}")
        gs, ws = B.stats(), P.stats()
        for key in ("attempts", "accepted", "crossings", "rays", "horizon", "escaped", "max_steps", "fp64_attempts"):
            assert gs[key] == ws[key], key
