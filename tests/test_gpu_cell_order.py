"""The order of references inside cells, against the oracle, where it can go
wrong: cells of every size class of the cell sort (one reference, up to 8, up
to 32, up to 256, more), with strands that follow one another in the index slab
(the task index alone breaks depth-key ties) and with strands whose index
ranges are shuffled (the full instance and segment key does), on both binning
backends. Every dump is compared exactly."""
import ctypes as C

import numpy as np
import pytest

from bevy_strand_rasterizer_b200 import abi
from bevy_strand_rasterizer_b200.plugin import pack_indexed_strands
from bevy_strand_rasterizer_b200.scene import CameraSpec
from common import build_scene, run_gpu, run_ref
from test_gpu_parity import _compare, _exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("backend", [0, 1])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("strands,points,side", [(300, 8, 160), (2500, 6, 64)])
def test_cell_order_matches_oracle(strands, points, side, shuffled, backend):
    scene = build_scene("tiny", strands=strands, points=points, width=side, height=side, dom=side,
                        settings_overrides={"fragment_counts_enabled": 1, "fine_binning_backend": backend,
                                            "ref_capacity_factor": 16})
    if shuffled:
        meta = scene.assets[0][0].meta
        meta["offset"] = np.random.default_rng(3).permutation(meta["offset"])
    if backend == 0 and not shuffled:
        p = run_gpu(scene)
        largest = int(p.dump(abi.DUMP_COUNTS).max())
        p.close()
        assert largest > 256 or side != 64
    _compare(scene)


@pytest.mark.parametrize("backend,n", [(0, 257), (0, 512), (0, 513), (0, 1024), (0, 1025), (1, 2048), (0, 2049), (0, 5000),
                                       (1, 8192), (0, 8193)])
def test_one_large_cell(n, backend):
    # n one-segment strands inside one cell: the merge sort's sizes and their
    # neighbours, up to the longest cell it takes and one more.
    scene = build_scene("tiny", cull=False, settings_overrides={"fine_binning_backend": backend, "ref_capacity_factor": 64})
    spec = CameraSpec(width=scene.camera_cfg.screen_width, height=scene.camera_cfg.screen_height, eye=(0.0, 0.0, 0.6))
    scene.cam.clip_from_world[:] = [float(x) for x in spec.clip_from_world()]
    scene.cam.world_position[:] = [float(x) for x in spec.eye]
    pos = np.zeros((n, 2, 3))
    pos[:] = 0.002 + np.random.default_rng(n).uniform(0.0, 2e-4, (n, 1, 3))
    pos[:, 1, 1] += 1e-4
    packed = pack_indexed_strands(pos.reshape(-1, 3).astype(np.float32), np.full(n, 2, np.uint32),
                                  np.arange(n, dtype=np.uint32) * 2, np.arange(n * 2, dtype=np.uint32))
    old = scene.assets[0][0]
    packed.aabb_min, packed.aabb_max = np.minimum(packed.aabb_min, old.aabb_min), np.maximum(packed.aabb_max, old.aabb_max)
    scene.assets[0] = (packed,) + scene.assets[0][1:]
    assert int(run_ref(scene).get(abi.DUMP_COUNTS).max()) == n
    _compare(scene)


@pytest.mark.parametrize("name,kw", [("tiny", {}), ("small", {}), ("small", dict(strands=20_000, width=1600, height=900))])
def test_pages_that_lose_their_references(name, kw):
    # A reference budget that runs out inside a group of pages: the pages kept,
    # flagged and listed are the oracle's, and the next frame with room for all
    # of them matches it everywhere.
    scene = build_scene(name, settings_overrides={"ref_capacity_factor": 1}, **kw)
    plugin, ref = run_gpu(scene), run_ref(scene)
    assert plugin.stats(allow_overflow=True).overflow_flags & 4
    for what in (abi.DUMP_PAGE_META, abi.DUMP_COUNTS, abi.DUMP_OFFSETS, abi.DUMP_ACTIVE_TILES, abi.DUMP_RUNS,
                 abi.DUMP_WORK):
        _exact(plugin.dump(what), ref.get(what), what)
    scene.settings.ref_capacity_factor = 16
    abi.check(plugin.lib.fiber_settings_set(plugin.ctx, C.byref(scene.settings)), "fiber_settings_set")
    run_gpu(scene, plugin=plugin)
    full = run_ref(scene)
    for what in (abi.DUMP_PAGE_META, abi.DUMP_REFS, abi.DUMP_WORK, abi.DUMP_DOM_OPACITY):
        _exact(plugin.dump(what), full.get(what), what)
    plugin.close()
