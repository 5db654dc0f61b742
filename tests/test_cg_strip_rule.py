"""The rule by which the corrected CG takes its on-chip form: with room for no block every image runs the streamed form;
with room for some, a launch never has more blocks than that, its borders fit their buffers, and the units cover the image."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "light-field-remote-vision_gb300" / "csrc"

SRC = r"""
#include <cstdio>
#include "cg_strip_rule.h"
using namespace lfrv;
int main() {
    long bad = 0, n = 0, taken = 0;
    const int caps[] = {0, 1, 15, 16, 17, 148, 152, 1000};
    for (int W = 2; W < 2200; W += 1 + W / 24)
        for (int H = 2; H < 2200; H += 1 + H / 24)
            for (int cap : caps) {
                const int R = strip_rows(W, H, cap);
                ++n;
                if (cap == 0) bad += R != 0;
                if (R == 0) continue;
                ++taken;
                const long units = (long)((W + kStripCols - 1) / kStripCols) * ((H + R - 1) / R);
                bad += R < 4 || R > kCgBatchMaxRows || !strip_fits(W, H, R) || strip_blocks(W, H, R) > cap;
                bad += (long)strip_blocks(W, H, R) * kStripUnits < units || units * 3 * strip_border(R) > 3L * W * H;
            }
    bad += strip_rows(1024, 1024, 152) != 28 || strip_rows(2048, 2048, 152) != 0 || strip_rows(64, 64, 152) != 4;
    std::printf("%ld %ld %ld\n", bad, n, taken);
    return 0;
}
"""


def test_rule(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(SRC)
    subprocess.run([cc, "-std=c++17", "-O1", f"-I{CSRC}", "-o", str(exe), str(src)], check=True)
    bad, n, taken = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and n > 10000 and taken > 10000
