"""Deep-opacity maps of materials whose opacity is not finite: an entry that
does not cover a pixel leaves its partial sums alone whatever its opacity."""
import numpy as np
import pytest

from bevy_strand_rasterizer_b200.plugin import StrandMaterial
from common import build_scene
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opacity", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("strands", [60, 300])
def test_non_finite_opacity(strands, opacity):
    # Two grooms in the same tiles, one of them with the default material.
    scene = build_scene("tiny", strands=strands, settings_overrides={"fragment_counts_enabled": 1, "ref_capacity_factor": 16})
    packed, _, place = scene.assets[0]
    moved = place.copy()
    moved[12:15] = (0.003, 0.002, -0.004)
    scene.assets.append((packed, StrandMaterial(absorption_color=(0.3, 0.6, 0.9, opacity), max_radius_pixels=3.0), moved))
    _compare(scene)
