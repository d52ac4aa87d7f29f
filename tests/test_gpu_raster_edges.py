"""The rasters against the oracle where their fast paths end: tile sizes other
than 8 x 8, strands that cross the near plane or pass behind the camera, radii
beyond the regular range, strands of repeated points and strands parallel to
the screen axes, rounds that are filled exactly, by one reference less and by
one more. Integer dumps and the deep-opacity maps are compared exactly."""
import numpy as np
import pytest

from bevy_strand_rasterizer_b200.plugin import FroxelConfig, StrandMaterial, pack_indexed_strands
from bevy_strand_rasterizer_b200.scene import CameraSpec
from common import build_scene
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu

SETTINGS = {"fragment_counts_enabled": 1, "ref_capacity_factor": 64}


def _camera(scene, **kw):
    spec = CameraSpec(width=scene.camera_cfg.screen_width, height=scene.camera_cfg.screen_height, **kw)
    scene.cam.clip_from_world[:] = [float(x) for x in spec.clip_from_world()]
    scene.cam.world_position[:] = [float(x) for x in spec.eye]


def _strands(scene, pos):
    """Replaces the scene's strands by polylines pos (strands, points, 3)."""
    n, m, _ = pos.shape
    packed = pack_indexed_strands(pos.reshape(-1, 3).astype(np.float32), np.full(n, m, np.uint32),
                                  np.arange(n, dtype=np.uint32) * m, np.arange(n * m, dtype=np.uint32))
    old = scene.assets[0][0]
    packed.aabb_min, packed.aabb_max = np.minimum(packed.aabb_min, old.aabb_min), np.maximum(packed.aabb_max, old.aabb_max)
    scene.assets[0] = (packed,) + scene.assets[0][1:]


@pytest.mark.parametrize("fx,fy", [(4, 4), (8, 4), (5, 7), (16, 8), (1, 64)])
def test_tile_sizes(fx, fy):
    scene = build_scene("tiny", width=150, height=110, settings_overrides=SETTINGS)
    scene.camera_cfg = FroxelConfig(150, 110, fx, fy, 16)
    scene.light_cfgs = [FroxelConfig(128, 128, fx, fy, 16)]
    _compare(scene)


@pytest.mark.parametrize("eye", [(0.0, 0.1, 0.2), (0.05, 0.3, 0.05), (0.0, -0.05, 0.12)])
def test_near_plane_and_behind(eye):
    scene = build_scene("tiny", settings_overrides=SETTINGS)
    _camera(scene, eye=eye, target=(0.02, 0.05, 0.0))
    _compare(scene)


@pytest.mark.parametrize("rmin,rmax", [(0.0, 0.0), (0.4, 12.0), (1.0, 3e18), (2e18, 2e18)])
def test_radii(rmin, rmax):
    scene = build_scene("tiny", material=StrandMaterial(min_radius_pixels=rmin, max_radius_pixels=rmax),
                        settings_overrides=SETTINGS)
    _compare(scene)


def test_repeated_points_and_axis_parallel_strands():
    scene = build_scene("tiny", settings_overrides=SETTINGS)
    _camera(scene, eye=(0.0, 0.0, 0.6))
    rng = np.random.default_rng(5)
    n, m = 200, 6
    pos = np.repeat(rng.uniform(-0.15, 0.15, (n, 1, 3)), m, axis=1)
    k = np.arange(m) * 0.01
    pos[0::4, :, 0] += k                     # along the screen's x
    pos[1::4, :, 1] += k                     # along its y
    pos[2::4, m // 2:, 1] += 0.03            # one long step, the rest repeated points
    pos[3::4, :, 2] -= k                     # away from the camera
    _strands(scene, pos)
    _compare(scene)


@pytest.mark.parametrize("strands", [127, 128, 129, 257])
def test_round_boundaries(strands):
    # One tile's worth of identical short strands: every reference of the tile
    # lies in a few cells, whose counts straddle the staged round.
    scene = build_scene("tiny", cull=False, settings_overrides=SETTINGS)
    _camera(scene, eye=(0.0, 0.0, 0.6))
    rng = np.random.default_rng(strands)
    pos = np.zeros((strands, 2, 3))
    pos[:, :, :2] = 0.001 + rng.uniform(0.0, 0.002, (strands, 1, 2))
    pos[:, 1, 1] += 0.001
    pos[:, :, 2] = rng.uniform(-0.05, 0.05, (strands, 1))
    _strands(scene, pos)
    _compare(scene)


@pytest.mark.parametrize("strands,light", [(255, 0), (256, 40), (513, 40), (6000, 1500)])
def test_heavy_and_light_runs(strands, light):
    # A clump of identical strands in a light tile (a heavy run, rounds of 256)
    # beside single ones. With 6000 the limit, 1 / 3552 of the references on the
    # 148 SMs of a B200, passes what the single ones leave in a tile: both rasters.
    scene = build_scene("tiny", cull=False, settings_overrides=SETTINGS)
    _camera(scene, eye=(0.0, 0.0, 0.6))
    rng = np.random.default_rng(strands + light)
    pos = np.zeros((strands + light, 2, 3))
    pos[:strands] = 0.001 + rng.uniform(0.0, 0.002, (strands, 1, 3))
    pos[strands:] = rng.uniform(-0.15, 0.15, (light, 1, 3))
    pos[:, 1, 1] += 0.001
    _strands(scene, pos)
    _compare(scene)


@pytest.mark.parametrize("strands,width,backend", [(1, 640, 0), (16, 640, 1), (33, 640, 0), (40, 96, 0), (700, 1280, 0)])
def test_segments_across_many_tiles(strands, width, backend):
    # Segments through the whole scene: more coarse tiles than a warp's queue
    # holds, tiles with more visits than its buffer, batches longer than its
    # stage; on a narrow screen, few tiles of many depth slices.
    scene = build_scene("tiny", cull=False, width=width, height=width // 2, settings_overrides=dict(SETTINGS, fine_binning_backend=backend))
    old = scene.assets[0][0]
    lo, hi = np.asarray(old.aabb_min, np.float64), np.asarray(old.aabb_max, np.float64)
    _strands(scene, np.random.default_rng(strands).uniform(lo, hi, (strands, 2, 3)))
    _compare(scene)


@pytest.mark.parametrize("scale", [1e-6, 1e13])
def test_scene_scale(scale):
    # 1e13: clip coordinates beyond the range of the projection's shared
    # reciprocal (w above 2^40); 1e-6: far below the near plane's distance.
    scene = build_scene("tiny", settings_overrides=SETTINGS)
    packed, material, m = scene.assets[0]
    m = m.copy()
    m[0] = m[5] = m[10] = scale
    scene.assets[0] = (packed, material, m)
    _camera(scene, eye=(0.0, 0.0, 0.6 * max(scale, 1.0)))
    _compare(scene)
