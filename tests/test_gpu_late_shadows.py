"""The wavefront form that traces an iteration's shadow rays beside the next one's extension rays, against the megakernel
and the barriered phases (stage timing). Films are the same bits: a contribution is the last addition to its sample in either form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(film):
    return np.concatenate([film.rgb.ravel(), film.lum_var.ravel()]).view(np.uint32)


# pools from the smallest (a slot renders many samples) to one slot per sample; depth 1 ends every path with its shadow ray pending;
# 129 and 513 samples leave part-filled tiles
@pytest.mark.parametrize("scene", ["cornell36", "icospheres"])
@pytest.mark.parametrize("w,h,spp,depth,pool", [(1, 1, 2, 8, 32), (43, 1, 3, 1, 32), (27, 19, 1, 8, 0), (171, 1, 3, 8, 0),
                                                (61, 37, 5, 8, 1000), (61, 37, 5, 1, 0), (64, 36, 4, 2, 2304)])
def test_late_shadow_rays_make_the_same_film(wfb, scene, w, h, spp, depth, pool):
    s = wfb.Scene.generate(scene, w, h, 1234, 16)
    p = wfb.RenderParams(spp=spp, seed=5, max_depth=depth, count_rays=True)
    mk, mst = wfb.GpuRenderer(s, wfb.MEGAKERNEL), wfb.RenderStats()
    want = mk.render(p, mst)
    r, st = wfb.GpuRenderer(s, wfb.WAVEFRONT), wfb.RenderStats()
    if pool:
        r.configure(paths_in_flight=pool)
    assert np.array_equal(_bits(r.render(p, st)), _bits(want))
    assert (st.extension_rays, st.shadow_rays) == (mst.extension_rays, mst.shadow_rays)
    assert np.array_equal(_bits(r.render(wfb.RenderParams(spp=spp, seed=5, max_depth=depth, stage_timing=True))), _bits(want))
    # sample ranges that do not start at 0, on a pool that has been used
    r.reset()
    r.run_passes(0, 1, p)
    if spp > 1:
        r.run_passes(1, spp - 1, p)
    assert np.array_equal(_bits(r.download(spp)), _bits(want))
