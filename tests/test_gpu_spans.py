"""fiber_span_times: a stage that ran has a time, one that did not has -1."""
import pytest

from bevy_strand_rasterizer_b200.plugin import StrandRasterizerPlugin
from common import build_scene, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backend", [0, 1])
def test_spans_follow_the_nodes(backend):
    scene = build_scene("tiny", settings_overrides={"fine_binning_backend": backend})
    p = run_gpu(scene)
    spans = p.span_times()
    assert spans.pop("strand_composite/composite") == -1.0
    assert min(spans.values()) >= 0.0
    total = spans.pop("frame/total")
    assert max(spans.values()) <= total
    p.close()
    # The prepass alone, in a context that has rendered nothing else: its nine
    # stages have their own ends.
    packed, material, place = scene.assets[0]
    p = StrandRasterizerPlugin(backend=backend)
    p.add_geometry(packed, material, place)
    p.frame_begin_raw(scene.camera_cfg, scene.cam, scene.light_cfgs, scene.lights_c)
    p.work_preparation_pass()
    spans = p.span_times()
    ran = {k for k, v in spans.items() if v >= 0.0}
    assert ran == {k for k in spans if k.startswith("strand_prepass/")} and len(ran) == 9
    p.close()
