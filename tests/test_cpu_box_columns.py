"""The register rows of a warp of box evaluation: every box in a column of its
own, the lanes without a box in columns that no box has (a shared column is
right only while its lanes stay in lockstep, which nothing enforces), every
row's offset within the 16 bits of a decoded instruction, and the whole within
the shared memory the kernel may ask for.  The layout is the header's own,
compiled for the host.  No device needed."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "temporalsetinversion_b200" / "csrc"

PROGRAM = r"""
#include <stdio.h>
#include "evalbox.h"

int main() {
  for (unsigned nregs = 4; nregs <= 256; ++nregs) {
    const unsigned per = tsi::narrow_boxes(nregs), cols = tsi::narrow_columns(nregs);
    if (per < 1 || per > 32 || nregs * cols * 8u > 65535u) return printf("offset: %u registers\n", nregs);
    if (tsi::narrow_bytes(nregs) < (size_t)(nregs + 1u) * cols * 8u + 512u) return printf("bytes: %u registers\n", nregs);
    if (tsi::narrow_bytes(nregs) > tsi::kNarrowMax) return printf("limit: %u registers\n", nregs);
    for (unsigned boxes = 1; boxes <= per; ++boxes) {
      unsigned owner[33] = {0};  // 1 + the lane of a box's column
      for (unsigned lane = 0; lane < 32; ++lane) {
        const unsigned c = tsi::narrow_column(nregs, lane);
        if (c >= cols) return printf("range: %u registers, lane %u\n", nregs, lane);
        if (lane < boxes) {
          if (owner[c]) return printf("shared: %u registers, lanes %u and %u\n", nregs, owner[c] - 1, lane);
          owner[c] = lane + 1;
        } else if (owner[c]) {
          return printf("spare lane in a box's column: %u registers, %u boxes, lane %u\n", nregs, boxes, lane);
        }
      }
    }
  }
  printf("ok\n");
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_no_two_lanes_share_a_live_column(tmp_path):
    cuda = next((d for d in ("/usr/local/cuda/include", "/usr/local/cuda/targets/x86_64-linux/include")
                 if (Path(d) / "cuda_runtime.h").exists()), None)
    if cuda is None:
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "columns.cpp", tmp_path / "columns"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", cuda, "-I", str(CSRC), "-I", str(CSRC.parents[1] / "include"), str(src),
                    "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.stdout.strip() == "ok", out.stdout
