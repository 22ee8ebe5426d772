"""Statistics of the wavefront's two-phase form (wavefront_late, the default of single renders with several samples) against
those of the barriered phases, which stage timing runs."""
import pytest

from test_ordered_traversal import _ball_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["cornell36", "icospheres"])
def test_stage_times_of_an_ordinary_render(wfb, scene):
    """Extension and shadow rays share a phase and are still told apart; the stages add up to no more than the kernel."""
    r = wfb.GpuRenderer(wfb.Scene.generate(scene, 128, 72, 1234, 16), wfb.WAVEFRONT)
    st = wfb.RenderStats()
    r.render(wfb.RenderParams(spp=8, seed=3, max_depth=8), st)
    assert st.stages["extend"] > 0 and st.stages["shadow"] > 0 and st.stages["classify"] > 0
    assert sum(st.stages.values()) <= st.render_ms


def test_queue_high_water_counts_the_last_bounce(wfb):
    """Two paths at a time through balls of every material: where the last bounce of a film is the only one of its material (the
    path ends in it), the material's high-water mark still counts it."""
    _, arrays = _ball_scene(wfb, 300, 3)
    r = wfb.GpuRenderer(wfb.Scene.from_arrays(dict(arrays, width=1, height=1)), wfb.WAVEFRONT)
    marks = {False: [], True: []}
    for seed in range(1, 301):
        for staged in marks:
            st = wfb.RenderStats()
            r.render(wfb.RenderParams(spp=2, seed=seed, max_depth=8, stage_timing=staged), st)
            marks[staged].append(tuple(st.queue_high_water[:3]))
    assert marks[False] == marks[True]
