"""Contexts created, rendered and closed on several host threads at once: the
first launches of a process configure the kernels, whichever thread they come
from, and a frame graph is captured while other threads register instances,
grow buffers and close contexts."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys, threading
sys.path[:0] = {paths!r}
import numpy as np, torch
from bevy_strand_rasterizer_b200 import abi
from common import build_scene, run_gpu
scene = build_scene("tiny", settings_overrides={{"history_enabled": 0, "dom_slices": 16}})
abi.load_library()
want = None
for _ in range(20):
    start, got = threading.Barrier(6), [None] * 6
    def work(k):
        stream = torch.cuda.Stream()
        start.wait()
        p = run_gpu(scene, fused=k % 2 == 1, stream=stream)
        got[k] = [p.dump(w).tobytes() for w in (abi.DUMP_REFS, abi.DUMP_DOM_OPACITY, abi.DUMP_COLOR)]
        p.close()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    want = want or got[0]
    assert want is not None and len(want[0]) > 0
    assert all(g == want for g in got)
print("same")
"""


def test_first_frames_on_six_threads():
    # A process of its own, so that no kernel was configured before.
    root = Path(__file__).resolve().parents[1]
    code = PROGRAM.format(paths=[str(root), str(root / "tests")])
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=240)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
