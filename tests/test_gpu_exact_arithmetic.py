"""The corrected reciprocals, quotients and square roots that the integer
stages and both rasters use in place of the general operators: equal to them
bit for bit over the ranges that their comments state (every reciprocal and
root of magnitude 2^-100 to 2^101, the quotients nearest to rounding
boundaries, seeded ones, every 16-bit and 24-bit unpacking)."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

from bevy_strand_rasterizer_b200 import build

pytestmark = pytest.mark.gpu

CHECKS = ("reciprocal", "square root", "near a boundary", "random", "unpacking")


def test_equal_to_the_operators(tmp_path):
    here = Path(__file__).resolve().parent
    lib = tmp_path / "exact_arithmetic.so"
    subprocess.run([build._nvcc(), *build.flags_for("fiber_raster.cu"), "-I", str(build.CSRC),
                    "-I", str(here.parent / "include"), "-shared", str(here / "exact_arithmetic.cu"), "-o", str(lib)],
                   check=True)
    out = (C.c_uint64 * (2 * len(CHECKS)))()
    assert C.CDLL(str(lib)).exact_arithmetic(out) == 0
    seen = {name: out[2 * k + 1] for k, name in enumerate(CHECKS)}
    assert seen["reciprocal"] == seen["square root"] == 2 * (201 << 23)
    assert seen["near a boundary"] > 100_000_000 and seen["random"] == 3 << 29 and seen["unpacking"] == 3 << 24
    assert {name: out[2 * k] for k, name in enumerate(CHECKS)} == dict.fromkeys(CHECKS, 0)
