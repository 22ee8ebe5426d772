"""The arm that the autotuner picks on a B200, where the two arms are far apart: a preview of the small scene, which the
megakernel renders in three quarters of the wavefront's time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tuner_picks_the_faster_arm_of_a_small_preview(wfb):
    w, h, spp = 320, 180, 16
    scene = wfb.Scene.generate("cornell36", w, h, 1234, 16)
    tuning = wfb.autotune(scene, w, h, probe_spp=8)
    ms = {}
    for mode in (wfb.MEGAKERNEL, wfb.WAVEFRONT):
        r = wfb.GpuRenderer(scene, mode)
        r.apply_tuning(tuning)
        times = []
        for _ in range(12):
            st = wfb.RenderStats()
            r.render(wfb.RenderParams(spp=spp, seed=3, max_depth=8), st)
            times.append(st.render_ms)
        ms[mode] = float(np.median(times))
    other = wfb.WAVEFRONT if tuning.mode == wfb.MEGAKERNEL else wfb.MEGAKERNEL
    assert ms[tuning.mode] < 1.1 * ms[other], (tuning.as_dict(), ms)
