"""Which parity says that the newest copy into an operand stage has landed (csrc/kernels/ring.h)."""
import os
import subprocess

import tnn_b200
from tnn_b200._build import CXX

KERNELS = os.path.join(os.path.dirname(tnn_b200.__file__), "csrc", "kernels")

PROGRAM = r"""
#include "ring.h"
#include <cstdio>
// A barrier that has completed `c` phases lets a wait for parity p through when c & 1 differs from p.
static bool passes(int c, unsigned p) { return (unsigned)(c & 1) != p; }
int main() {
  int checked = 0;
  for (int stages = 2; stages <= 8; ++stages)
    for (int copies = 1; copies <= 5 * stages; ++copies) {
      const int last = copies - 1, stage = last % stages;
      const unsigned phase = (last / stages) & 1;
      for (int s = 0; s < stages; ++s) {
        const int into = copies / stages + (s < copies % stages);  // copies that went into stage s
        const unsigned p = tnnb::ring_parity(s, stage, phase);
        if (!passes(into, p)) return 1;                  // all have landed
        if (into > 0 && passes(into - 1, p)) return 2;   // the newest is on its way
        ++checked;
      }
    }
  std::printf("%d", checked);
}
"""


def test_every_copy_is_waited_for(tmp_path):
    src, exe = tmp_path / "ring.cc", tmp_path / "ring"
    src.write_text(PROGRAM)
    subprocess.run([CXX, "-std=c++17", "-I", KERNELS, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and int(r.stdout) > 500


def test_rings_are_drained_as_a_whole():
    """No kernel settles for the newest copy of a ring, and the three that fetch tiles for their epilogue wait for those as well."""
    text = "".join(open(os.path.join(KERNELS, f)).read() for f in ("gemm_tcgen05.cu", "conv_implicit.cu"))
    assert "full[last" not in text and text.count("drain_stages(full") == 3
    assert text.count("epi_drain(ew, lane)") == 3
