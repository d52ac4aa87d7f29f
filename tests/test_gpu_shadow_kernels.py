"""Both kernels of the deep-opacity raster over the cases where they can go
wrong: every run as a light one, then every run as a heavy one, each compared
with the oracle. By the rule most small scenes have heavy runs alone."""
import ctypes as C

import numpy as np
import pytest

import test_gpu_opacity as opacities
import test_gpu_raster_edges as edges
from bevy_strand_rasterizer_b200 import abi
from bevy_strand_rasterizer_b200.plugin import StrandRasterizerPlugin
from common import build_scene, run_gpu
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu

LIGHT, HEAVY = 1, 2


def _heavy_runs(p, which=0):
    n = C.c_uint32()
    abi.check(p.lib.fiber_debug_shadow_kernel(p.ctx, which, C.byref(n)), "fiber_debug_shadow_kernel")
    return n.value


@pytest.fixture(params=[LIGHT, HEAVY], ids=["light", "heavy"])
def kernel(request, monkeypatch):
    """Every frame's shadow runs by one kernel; checks that it was that one."""
    which, begin, stats = request.param, StrandRasterizerPlugin.frame_begin_raw, StrandRasterizerPlugin.stats

    def begin_raw(self, *args, **kw):
        _heavy_runs(self, which)
        return begin(self, *args, **kw)

    def checked(self, *args, **kw):
        s = stats(self, *args, **kw)
        assert _heavy_runs(self, which) == (s.shadow_runs if which == HEAVY else 0)
        return s

    monkeypatch.setattr(StrandRasterizerPlugin, "frame_begin_raw", begin_raw)
    monkeypatch.setattr(StrandRasterizerPlugin, "stats", checked)


@pytest.mark.parametrize("fx,fy", [(4, 4), (5, 7), (16, 8), (1, 64)])
def test_tile_sizes(kernel, fx, fy):
    edges.test_tile_sizes(fx, fy)


@pytest.mark.parametrize("eye", [(0.0, 0.1, 0.2), (0.0, -0.05, 0.12)])
def test_near_plane_and_behind(kernel, eye):
    edges.test_near_plane_and_behind(eye)


@pytest.mark.parametrize("rmin,rmax", [(0.0, 0.0), (0.4, 12.0), (1.0, 3e18)])
def test_radii(kernel, rmin, rmax):
    edges.test_radii(rmin, rmax)


def test_repeated_points_and_axis_parallel_strands(kernel):
    edges.test_repeated_points_and_axis_parallel_strands()


@pytest.mark.parametrize("strands", [127, 128, 129, 255, 256, 257, 513])
def test_round_boundaries(kernel, strands):
    edges.test_round_boundaries(strands)


@pytest.mark.parametrize("slices", [1, 8, 16])
def test_slices(kernel, slices):
    _compare(build_scene("tiny", layers=slices, settings_overrides={"fragment_counts_enabled": 1, "ref_capacity_factor": 16}))


@pytest.mark.parametrize("opacity", [float("inf"), float("nan")])
def test_non_finite_opacity(kernel, opacity):
    opacities.test_non_finite_opacity(300, opacity)


@pytest.mark.parametrize("slices,blocks", [(4, 12), (12, 10), (16, 8)])
def test_rule(slices, blocks):
    # Half the references per resident block of the light runs' kernel, which
    # shared memory limits above 8 slices.
    import torch
    scene = build_scene("small", layers=slices, settings_overrides={"ref_capacity_factor": 8})
    p = run_gpu(scene)
    load = p.dump(abi.DUMP_RUNS)["load_score"][p.stats().camera_runs:].astype(np.uint64)
    share = np.float32(int(load.sum())) / np.float32(blocks * torch.cuda.get_device_properties(0).multi_processor_count)
    limit = int(max(np.float32(0.5) * share, np.float32(1.0)))
    heavy = int((load >= limit).sum())
    assert 0 < heavy < load.size
    assert _heavy_runs(p) == heavy
    p.close()
