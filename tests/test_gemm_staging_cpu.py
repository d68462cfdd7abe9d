"""Order of the GEMM epilogue's two staging boxes, on the CPU: the header that the kernel uses, compiled as plain C++."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "meshslice_b200" / "csrc"

# The epilogue's takes and sends for tiles of 256 columns of which `cols` are inside the matrix.  Stores are read in the
# order of sending; a wait leaves at most `left` of them unread, and the slowest copy engine reads nothing before a wait.
HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <deque>
#include "gemm/out_turn.h"
std::deque<int> unread;
msb::OutTurn turn{0};
int bad = 0;
int take(int taken) {
  while ((int)unread.size() > 1 - taken) unread.pop_front();
  const int box = turn.take();
  for (int u : unread) bad += u == box;
  return box;
}
void send(int box) { turn.sent(box); unread.push_back(box); }
int main(int, char** argv) {
  const bool dual = std::atoi(argv[1]), fp32 = std::atoi(argv[2]);
  const int cols = std::atoi(argv[3]);
  for (int tile = 0; tile < 5; ++tile) {
    int pre = -1, box = -1;
    for (int c = 0; c < 8; ++c) {
      if ((c & ~1) * 32 >= cols) continue;
      if (dual) {
        if ((c & 1) == 0) pre = take(0);
        else send(pre);
      }
      if (fp32) {
        if (c * 32 >= cols) continue;
        box = take(dual);
        bad += (c & 1) == 0 && box == pre;
        send(box);
      } else {
        if ((c & 1) == 0) { box = take(dual); bad += box == pre; }
        else send(box);
      }
    }
  }
  std::printf("%d\n", bad);
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("turn")
    (d / "main.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return d / "main"


@pytest.mark.parametrize("cols", [8, 24, 32, 40, 64, 72, 96, 136, 200, 224, 232, 256])
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("dual", [0, 1])
def test_no_box_is_written_while_its_store_is_unread(harness, dual, fp32, cols):
    out = subprocess.run([str(harness), str(dual), str(fp32), str(cols)], capture_output=True, text=True, check=True)
    assert out.stdout.strip() == "0"


def test_reduce_phase_refuses_a_misaligned_result():
    """The slot sums are written 16 bytes at a time; the refusal is the host's."""
    from meshslice_b200 import _native
    d = dict(M=256, N=256, K=64, A=1 << 20, B=1 << 20, lda=64, ldb=64, C=(1 << 20) + 8, ldc=256, red_n=2, red_work=1 << 20,
             red_slots=1 << 20, red_rows=256, red_cols=256, red_ld=256, status=1 << 20)
    with pytest.raises(RuntimeError, match="16-byte aligned C"):
        _native.load().gemm_run(d)
