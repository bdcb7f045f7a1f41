"""When a float64 grid set keeps face planes, compiled from the library's own header."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "his_gb300" / "csrc"
GB = 1 << 30


def test_face_planes_leave_a_caller_its_memory(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    (tmp_path / "rule.cpp").write_text(
        '#include <cstdio>\n#include <cstdlib>\n#include "face_rule.h"\n'
        "int main(int n, char** a) {\n"
        "    for (int i = 1; i + 2 < n; i += 3)\n"
        "        std::putchar(his::faces_taken(strtoull(a[i], 0, 10), strtoull(a[i + 1], 0, 10),"
        " strtoull(a[i + 2], 0, 10)) ? '1' : '0');\n}\n")
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(tmp_path / "rule.cpp"), "-o", str(tmp_path / "rule")], check=True)
    cells = 400 * 325
    planes = 80 * cells + 32 * 725
    cases = [
        ((planes, cells, 280 * GB), "1"),              # an empty device
        ((planes, cells, 16 * planes), "1"),           # the edge of a sixteenth
        ((planes, cells, 16 * planes - 1), "0"),
        ((planes, cells, 2 * planes), "0"),            # they would fit, and leave nothing
        ((planes, cells, 0), "0"),
        ((80 * 8100, 8100, 280 * GB), "0"),            # few cells
        ((80 * 39999, 39999, 280 * GB), "0"),
        ((80 * 40000, 40000, 280 * GB), "1"),
        ((4 * GB, 53_000_000, 280 * GB), "1"),
        ((4 * GB + 1, 53_000_000, 280 * GB), "0"),
        ((2 * GB, 26_000_000, 30 * GB), "0"),
    ]
    args = [str(v) for c, _ in cases for v in c]
    out = subprocess.run([str(tmp_path / "rule"), *args], check=True, capture_output=True, text=True).stdout
    assert out == "".join(w for _, w in cases)
