"""The plan of the marching heat kernel (lg_heat_plan.h) on the CPU: the planes
per CTA cost no more than the best of every chunk count, found in few tries,
and a tile that the grid fills costs less than one it does not."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "legendre_b200" / "csrc"

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include "lg_heat_plan.h"
using namespace lg;
static int64_t cost(int64_t tiles, int planes, int halo, int64_t slots, int zc) {
    return (tiles * ((planes + zc - 1) / zc) + slots - 1) / slots * (zc + 2 * halo + 4);
}
int main() {
    int wrong = 0;
    for (int64_t tiles : {1, 2, 7, 12, 100, 361, 5000})
        for (int planes : {1, 2, 3, 5, 97, 255, 256, 257, 512, 1001, 4000, 99991})
            for (int halo : {1, 2})
                for (int64_t slots : {148, 296, 592, 1184, 4736}) {
                    const int zc = march_planes(tiles, planes, halo, slots);
                    bool ok = zc >= 1 && zc <= std::min(planes, kMaxPlanes);
                    for (int chunks = (planes + kMaxPlanes - 1) / kMaxPlanes;
                         ok && chunks <= planes && tiles * (chunks - 1) <= 64 * slots; ++chunks) {
                        const int other = (planes + chunks - 1) / chunks;
                        ok = cost(tiles, planes, halo, slots, zc) <= cost(tiles, planes, halo, slots, other);
                    }
                    if (!ok && ++wrong < 5) std::printf("%ld tiles, %d planes: %d\n", (long)tiles, planes, zc);
                }
    // a search over every chunk count of these took above 20 ms
    const auto t = std::chrono::steady_clock::now();
    int sum = 0;
    for (int i = 0; i < 10; ++i) sum += march_planes(1, 1 << 30, 2, 1 << 26);
    const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count();
    // 8 cells of 8 or of 32 columns, the same threads and rows
    const int64_t narrow = 64, wide = 16;
    if (!(march_cost(narrow / 8, 512, march_planes(narrow / 8, 512, 2, 296), 2, 148, 2, 252, 4) <
          march_cost(wide * 2, 512, march_planes(wide * 2, 512, 2, 296), 2, 148, 2, 384, 2)))
        ++wrong;
    std::printf("%d wrong, %g s (%d)\n", wrong, s, sum);
    return wrong != 0 || s > 5e-3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_planes_per_cta(tmp_path):
    (tmp_path / "p.cpp").write_text(PROGRAM)
    exe = tmp_path / "p"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), str(tmp_path / "p.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
