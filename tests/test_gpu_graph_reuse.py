"""One context whose captured frame graph serves several frames: what a replay
must not keep of the frame it was captured for. Every fused frame is compared
with the oracle of its own scene."""
import ctypes as C

import numpy as np
import pytest

from bevy_strand_rasterizer_b200 import abi
from bevy_strand_rasterizer_b200.plugin import FroxelConfig
from common import build_scene, run_ref
from oracle_bridge import capacities, coarse_tiles
from test_gpu_parity import _exact

pytestmark = pytest.mark.gpu

DUMPS = (abi.DUMP_TASKS, abi.DUMP_PAGE_TABLE, abi.DUMP_PAGE_META, abi.DUMP_COUNTS, abi.DUMP_OFFSETS, abi.DUMP_REFS,
         abi.DUMP_ACTIVE_TILES, abi.DUMP_WORK, abi.DUMP_RUNS, abi.DUMP_DOM_DEPTH, abi.DUMP_DOM_OPACITY,
         abi.DUMP_SHADOW_MAP)


def _frames(scenes, order):
    """Renders scenes[k] for k in order in one context: the first frame node by
    node (it sizes the buffers and captures nothing), the others fused on one
    stream."""
    import torch
    from bevy_strand_rasterizer_b200.plugin import StrandRasterizerPlugin

    stream = torch.cuda.Stream()
    p = StrandRasterizerPlugin()
    abi.check(p.lib.fiber_settings_set(p.ctx, C.byref(scenes[0].settings)), "fiber_settings_set")
    for s in scenes:
        p.add_geometry(*s.assets[0])
    assets, refs = p.assets, [run_ref(s) for s in scenes]
    for n, k in enumerate(order):
        s, ref = scenes[k], refs[k]
        p.assets = [assets[k]]
        p._register()
        p.frame_begin_raw(s.camera_cfg, s.cam, s.light_cfgs, s.lights_c, stream)
        if n == 0:
            p.render_nodes(stream=stream)
        else:
            p.frame_fused(stream=stream)
        st, want = p.stats(), ref.stats()
        for name in ("binning_tasks", "allocated_pages", "fine_refs", "active_tiles", "work_items", "overflow_flags"):
            assert getattr(st, name) == getattr(want, name), f"frame {n}: {name}"
        for what in DUMPS:
            _exact(p.dump(what), ref.get(what), what)
        color, ref_color = p.dump(abi.DUMP_COLOR).astype(np.float32), ref.get(abi.DUMP_COLOR).astype(np.float32)
        assert float(np.max(np.abs(color - ref_color))) <= 2e-3, f"frame {n}: colour"
    p.close()


def test_fine_tiles_grow_under_a_reused_graph():
    # With 148 SMs 60,000 strands of two frusta take 1,876 look-back tiles of
    # the fine prepass, 19,200 take 600 (64 strands each) and 18,000 take 1,126
    # (32 each): the third frame replays the graph captured for the second.
    scenes = [build_scene("tiny", strands=n, points=4, cull=False,
                          settings_overrides={"history_enabled": 0, "ref_capacity_factor": 16})
              for n in (60_000, 19_200, 18_000)]
    _frames(scenes, [0, 1, 2])


@pytest.mark.parametrize("backend", [0, 1])
def test_work_items_grow_under_a_reused_graph(backend):
    # The third frame replays the graph captured for 300 strands and has more
    # work items than a frame of 300 strands has room for.
    scenes = [build_scene("tiny", strands=n, points=m, width=320, height=240, dom=256, cull=False,
                          settings_overrides={"history_enabled": 0, "ref_capacity_factor": 8,
                                              "fine_binning_backend": backend}) for n, m in ((6_000, 16), (300, 4))]
    cfgs = [c.to_c() for c in [scenes[1].camera_cfg] + scenes[1].light_cfgs]
    room = capacities(300 * 3, 300, 2, coarse_tiles(cfgs), scenes[1].settings).work_capacity
    assert run_ref(scenes[0]).stats().work_items > room
    _frames(scenes, [0, 1, 0])


def test_dom_size_under_a_reused_graph():
    # 256^2 maps in 4 px tiles and 512^2 maps in 8 px tiles have the same coarse
    # tiles; the third frame has four deep-opacity pages where the second had one.
    scenes = [build_scene("tiny", dom=dom, settings_overrides={"history_enabled": 0, "dom_page_pool": 8})
              for dom in (512, 256)]
    scenes[1].light_cfgs = [FroxelConfig(256, 256, 4, 4, 16)]
    _frames(scenes, [0, 1, 0])
