"""Statistics of the wavefront's two-phase form (wavefront_late, the default of single renders with several samples) against
those of the barriered phases, which stage timing runs."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["cornell36", "icospheres"])
def test_stage_times_of_an_ordinary_render(wfb, scene):
    """Extension and shadow rays share a phase and are still told apart; the stages add up to no more than the kernel."""
    r = wfb.GpuRenderer(wfb.Scene.generate(scene, 128, 72, 1234, 16), wfb.WAVEFRONT)
    st = wfb.RenderStats()
    r.render(wfb.RenderParams(spp=8, seed=3, max_depth=8), st)
    assert st.stages["extend"] > 0 and st.stages["shadow"] > 0 and st.stages["classify"] > 0
    assert sum(st.stages.values()) <= st.render_ms
