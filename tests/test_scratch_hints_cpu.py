"""How far the buffers of a batch's workers grow beyond their own needs (csrc/hints.hpp), compiled for the host."""

from __future__ import annotations

import os
import subprocess

from conftest import PKG

PROGRAM = r"""
#include <cassert>
#include <vector>
#include "hints.hpp"
using sdfgpu::ScratchHints;
int main() {
  ScratchHints H;
  struct Buf { std::size_t cap = 0, slack = 0; };
  std::vector<Buf> bufs(8 * 40);  // 8 workers with 40 buffers each
  unsigned rng = 1;
  std::size_t own = 0, all = 0;
  for (int item = 0; item < 400; ++item) {  // items of 1 MB to 100 MB a buffer reach the workers in any order
    rng = rng * 1664525u + 1013904223u;
    const int worker = (rng >> 8) % 8;
    const std::size_t need = (std::size_t)(1 + (rng >> 16) % 100) << 20;
    for (int b = 0; b < 40; ++b) {
      Buf& q = bufs[worker * 40 + b];
      if (q.cap >= need) continue;
      H.give_back(q.slack);
      const std::size_t want = need + need / 8, got = H.grant("b" + std::to_string(b), need, want);
      assert(got >= want && got <= std::max(want, ScratchHints::kHintMax + ScratchHints::kHintMax / 8));
      q = {got, got - want};
    }
    own = all = 0;
    for (const Buf& q : bufs) { all += q.cap; own += q.cap - q.slack; }
    assert(all - own == H.slack && H.slack <= ScratchHints::kSlackMax);
  }
  assert(all - own > 0);  // it does grow them
}
"""


def test_workers_slack_is_bounded(tmp_path):
    src, exe = tmp_path / "hints.cpp", tmp_path / "hints"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(PKG, "csrc"), str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
