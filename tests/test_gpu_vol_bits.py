"""One ray, one result: the volumetric kernels (spectral FP64, its mixed form and
its batched form; RGB FP64 and mixed; the debug trace) give the same bits for
the same sample, at spins whose rays pass through the plunging region inside
the innermost stable orbit and one without rotation."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 40, 36
SCENES = [(0.0, 60.0), (0.3, 25.0), (0.5, 60.0), (0.7, 85.0), (0.9, 60.0), (0.95, 20.0)]


def scene(grrt, spin, incl):
    p = grrt.config_params(3, width=W, height=H, spin=spin, observer_theta=math.radians(incl),
                           disk_seed=int(100 * spin + incl))
    if spin == 0.0:
        p.update(metric_type=grrt.METRIC_SCHWARZSCHILD)
    return p


@pytest.mark.parametrize("spin,incl", SCENES)
def test_spectral_forms_agree_to_the_bit(grrt, need_gpu, spin, incl):
    import torch
    bins = [grrt.log_bins(n=9), grrt.log_bins(n=33)]
    cams = [scene(grrt, spin, incl) for _ in bins]
    got = grrt.Batch(cams, freqs=bins).render_spectral()
    for p, f, batch in zip(cams, bins, got):
        R = grrt.Renderer(p, freqs=f)
        cube = {}
        for form in (grrt.FORM_FP64, grrt.FORM_MIXED):
            R.set_precision(form)
            buf = torch.full((H, W, len(f)), float("nan"), dtype=torch.float64, device="cuda")
            R.render_spectral_device(buf, W, H)
            torch.cuda.synchronize()
            cube[form] = buf.cpu().numpy()
        assert (cube[grrt.FORM_FP64] > 0).any()
        np.testing.assert_array_equal(cube[grrt.FORM_MIXED], cube[grrt.FORM_FP64])
        np.testing.assert_array_equal(batch, cube[grrt.FORM_FP64])


@pytest.mark.parametrize("spin,incl", SCENES)
def test_rgb_forms_and_debug_trace_agree_to_the_bit(grrt, need_gpu, spin, incl):
    import torch
    from oracle_bind import jittered_samples
    R = grrt.Renderer(scene(grrt, spin, incl))
    rgb = {}
    for form in (grrt.FORM_FP64, grrt.FORM_MIXED):
        R.set_precision(form)
        buf = torch.full((H * W, 3), float("nan"), dtype=torch.float64, device="cuda")
        R.render_device(None, buf, None)
        torch.cuda.synchronize()
        rgb[form] = buf.cpu().numpy()
    want = rgb[grrt.FORM_FP64]
    assert (want > 0).any()
    np.testing.assert_array_equal(rgb[grrt.FORM_MIXED], want)
    pix = np.nonzero(want.any(axis=1))[0][::17]
    xs, ys = jittered_samples(W, H, 1, pix)
    for p, x, y in zip(pix, xs, ys):
        np.testing.assert_array_equal(R.debug_trace(x, y)[-1]["v"][3:6], want[p], err_msg=f"pixel {p}")
