"""Device memory kept by a host thread between calls belongs to the context it
was allocated in.

CPU: a C++ program runs the keeping rule against a counting allocator: the same
context uses its block again, another context never sees or frees it, and a
thread that ends frees what is still alive.
GPU: byte features before and after a device reset, in a process of its own.
"""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include <map>
#include <set>
#include "kept_block.h"
// contexts by device; 0 = none. live: address -> context it was made in
static std::map<int, uint64_t> ctx_of;
static int dev;
static uint64_t now;
static std::map<void*, uint64_t> live;
static size_t next = 0x1000;
static int fail;
struct Fake {
  uint64_t context() { return now; }
  void init() { now = ctx_of[dev]; }
  int device() { return dev; }
  void set_device(int d) { dev = d, now = ctx_of[d]; }
  int alloc(void** p, size_t bytes) {
    if (fail) return 2;
    *p = reinterpret_cast<void*>(next += 0x1000);
    live[*p] = now;
    return 0;
  }
  void free(void* p) {
    if (!live.count(p) || live[p] != now) printf("foreign or dead block freed\n"), exit(1);
    live.erase(p);
  }
};
static void reset(int d) {  // destroys the device's context and its memory
  for (auto i = live.begin(); i != live.end();) i = i->second == ctx_of[d] ? live.erase(i) : std::next(i);
  ctx_of[d] += 100;
  if (dev == d) now = 0;
}
#define NEED(c) do { if (!(c)) return printf("line %d: %s\n", __LINE__, #c), 1; } while (0)
int main() {
  ctx_of[0] = 1, ctx_of[1] = 2;
  void *a, *b, *c;
  bool mine;
  {
    ngap::KeptBlocks<Fake> k;
    dev = 0, now = 0;  // nothing current yet
    NEED(k.reserve(100, 1000, &a, &mine) == 0 && !mine && live[a] == 1);
    NEED(k.reserve(60, 1000, &b, &mine) == 0 && !mine && b == a && live.size() == 1);   // same context keeps
    NEED(k.reserve(200, 1000, &b, &mine) == 0 && !mine && b != a && live.size() == 1);  // grows: one block
    NEED(k.reserve(2000, 1000, &c, &mine) == 0 && mine && c != b && live.size() == 2);  // too large to keep
    Fake().free(c);
    Fake().set_device(1);  // another device's context: a block of its own, the first stays
    NEED(k.reserve(100, 1000, &c, &mine) == 0 && !mine && live[c] == 2 && live.size() == 2);
    Fake().set_device(0);
    NEED(k.reserve(100, 1000, &a, &mine) == 0 && !mine && a == b);
    now = 77;  // another context of the same device, made by the caller
    NEED(k.reserve(100, 1000, &a, &mine) == 0 && !mine && a != b && live[a] == 77);
    now = ctx_of[0];
    NEED(k.reserve(100, 1000, &a, &mine) == 0 && !mine && a == b);
    reset(0);  // the block is gone: it is neither used nor freed again
    live[b] = 5;  // its address now belongs to somebody else
    NEED(k.reserve(100, 1000, &a, &mine) == 0 && !mine && a != b && live[a] == 101 && live[b] == 5);
    live.erase(b);
    for (int i = 0; i < 6; i++) {  // more contexts than are remembered: not kept, the caller frees
      reset(0);
      NEED(k.reserve(100, 1000, &a, &mine) == 0 && live[a] == now);
      if (mine) Fake().free(a);
    }
    NEED(mine);
    Fake().set_device(1);
    fail = 1;
    NEED(k.reserve(500, 1000, &a, &mine) == 2 && a == nullptr);  // the small block was given back
    NEED(live.empty() || (live.size() == 1 && live.begin()->second == 77));
    fail = 0;
    NEED(k.reserve(500, 1000, &a, &mine) == 0 && live[a] == 2);
    Fake().set_device(0);
  }
  // the thread ended with device 0 current: device 1's block was freed too, the
  // block of the context that the caller made is left to it
  NEED(live.size() == 1 && live.begin()->second == 77);
  printf("ok\n");
  return 0;
}
"""


def test_blocks_stay_in_their_context(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "check.cpp").write_text("#include <cstdlib>\n" + CHECK)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "ngap_b200", "csrc"),
                    str(tmp_path / "check.cpp"), "-o", str(tmp_path / "check")], check=True)
    r = subprocess.run([str(tmp_path / "check")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


RESET = r"""
import ctypes
import numpy as np
import ngap_b200 as nb
from ngap_b200 import cost_model as cm

nb.lib()
cuda = ctypes.CDLL("libcuda.so.1")
rt = next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l)
rt = ctypes.CDLL(rt)  # the runtime the library uses


def context_id():
    i = ctypes.c_ulonglong()
    assert cuda.cuCtxGetId(None, ctypes.byref(i)) == 0
    return i.value


rng = np.random.default_rng(2)
data = rng.integers(0, 9, size=100000).astype(np.uint8)
args = (np.array([0, 5, 50000]), np.arange(3), np.zeros(3, np.int64), np.array([1, 700, 30001]))
want = cm.byte_features(data, *args)
ids = [context_id()]
for _ in range(6):
    assert np.array_equal(cm.byte_features(data, *args), want)
    assert rt.cudaDeviceReset() == 0
    assert np.array_equal(cm.byte_features(data, *args), want)
    ids.append(context_id())
assert len(set(ids)) == len(ids), ids
print("ok")
"""


@pytest.mark.gpu
def test_features_after_a_device_reset(built):
    r = subprocess.run([sys.executable, "-c", RESET], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
