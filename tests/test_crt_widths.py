"""Register widths of the FP64 form's CRT (csrc/crt_widths.cuh) on the CPU: every word count has a width of
at least its words and, above eight, of less than twice as many."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sdpx.rs_b200" / "csrc"
SRC = r"""
#include <cstdio>
#include "crt_widths.cuh"
int main() {
  for (int w = 1; w <= sdpxg::kCrtMaxWords; ++w) std::printf("%d\n", sdpxg::crt_f64_words(w));
}
"""


def test_widths_fit(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "w.cc").write_text(SRC)
    subprocess.run([gxx, "-std=c++17", "-I", str(CSRC), str(tmp_path / "w.cc"), "-o", str(tmp_path / "w")], check=True)
    got = [int(v) for v in subprocess.run([tmp_path / "w"], capture_output=True, text=True).stdout.split()]
    assert len(got) == 64
    for words, width in enumerate(got, 1):
        assert words <= width <= max(8, 2 * words - 1)
