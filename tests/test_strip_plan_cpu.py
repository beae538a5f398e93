"""The fixed unit heights of the FP32 batched step (lg_strip_plan.h), on the CPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "legendre_b200" / "csrc"

# blocks, strips a block, rows of a block -> rows a unit, on 148 SMs
HEIGHTS = [(16, 1, 24, 8), (8, 2, 64, 8), (32, 2, 64, 8), (128, 2, 64, 8), (432, 2, 48, 8), (1024, 2, 64, 8),
           (4096, 2, 64, 32), (2048, 2, 64, 16), (1500, 3, 50, 12), (12, 1, 20, 8), (100, 1, 7, 4), (100, 1, 3, 3),
           (100, 1, 1, 1), (100000, 1, 16, 16), (100000, 8, 256, 32)]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_batched_heights(tmp_path):
    calls = "".join('std::printf("%%d\\n", lg::strip_batch_rows_f32(%d, %d, %d, 148));' % h[:3] for h in HEIGHTS)
    (tmp_path / "h.cpp").write_text('#include <cstdio>\n#include "lg_strip_plan.h"\nint main() {%s}' % calls)
    exe = tmp_path / "h"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(tmp_path / "h.cpp"), "-o", str(exe)], check=True)
    got = [int(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    assert got == [h[3] for h in HEIGHTS]
