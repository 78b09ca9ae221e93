"""Publications of the dataflow Cholesky's chain (csrc/chol_publish.cuh) on the CPU: the chain and every
tile item of the real work list run as far ahead as their inputs let them, and only then does the
publishing warp look at its barrier.  A parity wait sees phase q of a barrier after c completions when
c and q differ in parity, so it must never be two behind."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "sdpx.rs_b200" / "csrc"

HARNESS = r"""
#include <cstdio>
#include <vector>
#include "chol_publish.cuh"
#include "engine.cuh"
using namespace sdpxg;
static int replay(int nt) {
  const std::vector<unsigned> items = chol_schedule(nt);
  std::vector<int> prog(nt, 0), pre_d(nt, 0), pre_o(nt, 0);
  std::vector<char> done(items.size(), 0);
  std::vector<int> completions(chol_publish::kSlots, 0);
  int arrived = 0, published = 0;  // publications the chain has arrived for / that are out
  const int total = 2 * nt - 1;
  for (;;) {
    bool moved = false;
    for (size_t t = 1; t < items.size(); ++t) {  // the tiles of U: their inputs as the kernel waits for them
      const unsigned type = items[t] >> 30;
      const int k = (int)((items[t] >> 20) & 1023u), i = (int)((items[t] >> 10) & 1023u), j = (int)(items[t] & 1023u);
      if (done[t] || type == kCholInv || prog[i] < k || prog[j] < k) continue;
      if (type == kCholFull) {
        if (prog[i] < i + 1) continue;
        prog[j] = i + 1;
      } else {
        (i == j ? pre_d : pre_o)[i] = 1;
      }
      done[t] = 1;
      moved = true;
    }
    if (arrived < total) {  // the chain's next step: it waits for the PRE tiles alone
      const int k = arrived / 2;
      if (arrived & 1 ? k == 0 || pre_o[k] : k < 2 || pre_d[k]) {
        ++completions[chol_publish::slot(arrived)];
        ++arrived;
        moved = true;
      }
    }
    if (moved) continue;
    if (published == total) return 0;
    int phase = 0;  // of publication `published` on its barrier
    for (int t = 0; t < published; ++t) phase += chol_publish::slot(t) == chol_publish::slot(published);
    if ((phase & 1) != chol_publish::parity(published)) return 1;
    if ((completions[chol_publish::slot(published)] & 1) == (phase & 1)) return 2;  // it waits for good
    const int k = published / 2;
    if (published & 1) prog[k + 1] = k + 1;
    else prog[k] = k + 1;
    ++published;
  }
}
int main() {
  for (int nt = 1; nt <= 40; ++nt) {
    const int rc = replay(nt);
    if (rc) { std::printf("nt=%d: %d\n", nt, rc); return 1; }
  }
  std::printf("ok\n");
  return 0;
}
"""


def test_no_publication_is_missed(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not pathlib.Path(nvcc).exists():
        pytest.skip("nvcc not available")
    src = tmp_path / "pub.cu"
    src.write_text(HARNESS)
    exe = tmp_path / "pub"
    subprocess.run([nvcc, "-std=c++17", "-O1", f"-I{CSRC}", str(src), "-o", str(exe)], check=True,
                   capture_output=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
