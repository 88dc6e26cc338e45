"""Slices of scanned pieces: their candidate and run buffers stay within 64 and
256 MB at the shortest and the longest runs, and cover the pieces in order."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include "slices.h"
using namespace ngap;
#define NEED(c) do { if (!(c)) return printf("line %d: %s (run_len %d)\n", __LINE__, #c, rl), 1; } while (0)
int main(int argc, char** argv) {
  const int rl = atoi(argv[1]);
  for (int len : {256, 512, 4096})
    for (int64_t total : {(int64_t)len, (int64_t)len * 3 + 17, (int64_t)100 << 20}) {
      std::vector<PieceDev> pieces[2];
      const std::vector<int32_t> run_len = {rl, 64};
      for (int64_t at = 0; at < total; at += len) {
        PieceDev p{};
        p.lo = (uint32_t)at;
        p.hi = (uint32_t)std::min<int64_t>(at + len, total);
        p.tile = 0;
        pieces[0].push_back(p);
        p.tile = (at / len) & 1;
        pieces[1].push_back(p);
      }
      int64_t cands = 0, runs = 0;
      const std::vector<Slice> s = make_slices(pieces, run_len, &cands, &runs);
      NEED(cands * 2 <= 64 << 20 && runs * (int64_t)sizeof(RunDev) <= 256 << 20);
      int32_t next = 0;
      for (size_t k = 0; k < s.size(); k++) {
        NEED(s[k].begin == next && s[k].count > 0);
        next += s[k].count;
        int64_t pos = 0, r = 0;
        for (int32_t i = s[k].begin; i < next; i++) {
          const bool layered = i >= (int32_t)pieces[0].size();
          const PieceDev& p = layered ? pieces[1][i - pieces[0].size()] : pieces[0][i];
          NEED(layered == s[k].layered);
          NEED(s[k].one_tile < 0 || s[k].one_tile == p.tile);
          const int64_t n = p.hi - p.lo;
          pos += n;
          // every position a candidate, and a run for start-of-data states alone
          r += std::max<int64_t>((n + run_len[p.tile] - 1) / run_len[p.tile], 1);
          NEED(n <= s[k].longest);
        }
        NEED(pos <= cands && r <= s[k].runs && s[k].runs <= runs);
      }
      NEED(next == (int32_t)(pieces[0].size() + pieces[1].size()));
      // a batch of the same positions reserves at least that
      BatchShape b;
      b.tiles = b.scanned = 2;
      b.run_len = std::min(rl, 64);
      b.positions = total;
      b.streams = 1;
      b.chunk = len;
      b.warps = 4736;
      const PlanRoom room = plan_room(b);
      NEED(room.cands >= cands && room.runs >= runs && room.pieces >= next);
    }
  return 0;
}
"""


@pytest.mark.parametrize("run_len", [4, 5, 16, 64])
def test_slices_stay_within_their_buffers(tmp_path, run_len):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(cuda, "include", "vector_types.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    (tmp_path / "check.cpp").write_text(CHECK)
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "ngap_b200", "csrc"),
                    "-I", os.path.join(cuda, "include"), str(tmp_path / "check.cpp"), "-o",
                    str(tmp_path / "check")], check=True)
    r = subprocess.run([str(tmp_path / "check"), str(run_len)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
