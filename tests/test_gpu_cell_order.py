"""The order of references inside cells, against the oracle, where it can go
wrong: cells of every size class of the cell sort (one reference, up to 8, up
to 32, up to 256, more), with strands that follow one another in the index slab
(the task index alone breaks depth-key ties) and with strands whose index
ranges are shuffled (the full instance and segment key does), on both binning
backends. Every dump is compared exactly."""
import numpy as np
import pytest

from bevy_strand_rasterizer_b200 import abi
from common import build_scene, run_gpu
from test_gpu_parity import _compare

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
