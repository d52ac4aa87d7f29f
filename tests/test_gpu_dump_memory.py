"""fiber_dump of the references, which the device holds as task indices: it
needs no device memory of its own, and a dump between two nodes leaves the
frame as it is."""
import numpy as np
import pytest

from bevy_strand_rasterizer_b200 import abi
from common import build_scene, run_gpu, run_ref

pytestmark = pytest.mark.gpu


def test_dump_on_a_full_device():
    import torch
    scene = build_scene("small", strands=20_000, settings_overrides={"history_enabled": 0, "ref_capacity_factor": 8})
    p = run_gpu(scene)
    want = p.dump(abi.DUMP_REFS).copy()
    assert want.nbytes > 24 << 20
    hold = []
    for size in (1 << 30, 1 << 24):  # all but some 16 MB of the device
        while torch.cuda.mem_get_info()[0] > size + (1 << 24):
            n = (torch.cuda.mem_get_info()[0] - (1 << 24)) // size * size
            hold.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
    try:
        got = p.dump(abi.DUMP_REFS)
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)
    p.close()


@pytest.mark.parametrize("backend", [0, 1])
def test_dump_between_the_nodes(backend):
    scene = build_scene("tiny", settings_overrides={"history_enabled": 0, "fine_binning_backend": backend})
    p = run_gpu(scene)
    color, opacity = p.dump(abi.DUMP_COLOR).copy(), p.dump(abi.DUMP_DOM_OPACITY).copy()
    p.frame_begin_raw(scene.camera_cfg, scene.cam, scene.light_cfgs, scene.lights_c)
    p.work_preparation_pass()
    refs = p.dump(abi.DUMP_REFS)
    p.strand_shadow_rasterizer_pass()
    p.strand_shading_pass()
    p.strand_rasterizer_pass()
    assert np.array_equal(refs, run_ref(scene).get(abi.DUMP_REFS))
    assert np.array_equal(p.dump(abi.DUMP_REFS), refs)
    for what, v in ((abi.DUMP_COLOR, color), (abi.DUMP_DOM_OPACITY, opacity)):
        assert np.array_equal(p.dump(what).view(np.uint8), v.view(np.uint8))
    p.close()
