"""Which device inputs are read in place: memory of the engine's own GPU only.

CPU: the rule, compiled against made-up pointer attributes. GPU: pinned host
memory handed over as device memory is copied, and gives the oracle's reports.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include "plan_rules.h"
using namespace ngap;
int main() {
  int asked = 0;
  auto at = [&](uintptr_t address, bool on_device, uint64_t bytes, bool device, int owner, int engine) {
    return reads_in_place(reinterpret_cast<const void*>(address), on_device, bytes, engine, [&](const void*) {
      asked++;
      return InputMemory{device, owner};
    });
  };
  // the engine's own GPU, aligned; another GPU either way; host or managed memory
  const bool own[] = {at(0x100, true, 64, true, 0, 0), at(0x100, true, 64, true, 3, 3)};
  const bool other[] = {at(0x100, true, 64, true, 1, 0), at(0x100, true, 64, true, 0, 1),
                        at(0x100, true, 64, false, 0, 0), at(0x100, true, 64, false, -1, 0)};
  const int before = asked;
  // no question about what is copied anyway
  const bool copied[] = {at(0x101, true, 64, true, 0, 0), at(0x108, true, 64, true, 0, 0),
                         at(0x100, true, 65, true, 0, 0), at(0x100, true, 0, true, 0, 0),
                         at(0x100, false, 64, true, 0, 0)};
  for (bool b : own) if (!b) return printf("own memory is copied\n"), 1;
  for (bool b : other) if (b) return printf("memory elsewhere is read in place\n"), 1;
  for (bool b : copied) if (b) return printf("unaligned or host input is read in place\n"), 1;
  return before == 6 && asked == 6 ? 0 : 1;
}
"""


def test_only_the_engines_own_memory_is_read_in_place(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "check.cpp").write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "ngap_b200", "csrc"),
                    str(tmp_path / "check.cpp"), "-o", str(tmp_path / "check")], check=True)
    r = subprocess.run([str(tmp_path / "check")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


class AsDevice:
    """Pinned host memory handed over as device memory (the address is valid there)."""

    is_cuda = True

    def __init__(self, tensor):
        self.tensor = tensor

    def data_ptr(self):
        return self.tensor.data_ptr()

    def numel(self):
        return self.tensor.numel()

    def element_size(self):
        return 1


@pytest.mark.gpu
def test_pinned_memory_as_device_input(engine):
    import torch
    anml, data = W.literal_set(seed=5, n_patterns=20, input_len=200_016, plant_every=997)
    groups = nb.Groups(nb.Nfa.from_string(anml), group_num=1)
    tables = nb.Tables(groups, precompute_depth=2)
    want, _ = oracle.match(groups.views(), data, 1, len(data))
    buf = AsDevice(torch.from_numpy(data.copy()).pin_memory())
    assert len(want) and np.array_equal(engine.match(tables, buf, 1, len(data)), want)
