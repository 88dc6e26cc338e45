"""The host side of a match on the CPU, against a stand-in for the CUDA runtime
(fake_cudart.c): what is launched and uploaded after an allocation has failed,
and after buffers have moved. Each check runs in a process of its own."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = r"""
import ctypes
import numpy as np
import ngap_b200 as nb
from ngap_b200 import workloads as W
from ngap_b200._lib import lib

fake = ctypes.CDLL(None)
size = lambda name: ctypes.c_size_t.in_dll(fake, name)
count = lambda name: ctypes.c_long.in_dll(fake, name).value


def log(f, *a, **kw):
    "Launches and asynchronous copies of one call."
    fake.fake_reset()
    f(*a, **kw)
    return (ctypes.c_char * (1 << 20)).in_dll(fake, "fake_log").value.decode().split(";")[:-1]


def fails(f, *a, **kw):
    try:
        f(*a, **kw)
    except nb.NgapError as ex:
        assert ex.status == 5 and "out of memory" in str(ex), ex
        return
    raise AssertionError("the allocation did not fail")


def tables(text, depth=2, groups=1):
    return nb.Tables(nb.Groups(nb.Nfa.from_string(text), group_num=groups), precompute_depth=depth)


CAP = 4096
"""


@pytest.fixture(scope="module")
def run(built, tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("gcc") is None or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime_api.h")):
        pytest.skip("no C compiler or CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", so], check=True)

    def go(body):
        r = subprocess.run([sys.executable, "-c", PRELUDE + body + "\nprint('ok')"], cwd=ROOT, timeout=300,
                           env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True)
        assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
    return go


FAILED_PLAN = r"""
text, _ = W.literal_set(seed=5, n_patterns=20, input_len=1000, plant_every=100)
t = tables(text)
ts = nb.TableSet([t])
short, long = np.zeros(3000, np.uint8), np.zeros(9_000_000, np.uint8)


def plain(e, data):
    e.match_async(t, data, 1, len(data), result_capacity=CAP)


def batch(e, data):
    n = len(data) // 3
    nb.batch_match_async(e, ts, data, [0, n, 2 * n], [n, n, n], [0, 0, 0], result_capacity=CAP)


for first in (plain, batch):
    for other in (plain, batch):
        e = nb.Engine(0)
        want = log(first, e, short)
        assert any("match_kernel" in x for x in want) and not any("scan_kernel" in x for x in want)
        again = log(first, e, short)  # the plan is kept: nothing to upload but the input
        assert len(again) < len(want)
        # the longer plan's candidate list (2 bytes a position) cannot be had
        # (the input is copied into a buffer of half that size)
        size("fake_fail_at").value = 2 * len(long) - 4096
        fails(other, e, long)
        size("fake_fail_at").value = 0
        # the first call again: its own units are uploaded and launched, not the other plan's
        assert log(first, e, short) == want
        # and the longer input goes through once there is room
        assert any("scan_kernel" in x for x in log(other, e, long))
        assert log(first, e, short) == want
"""


def test_failed_plan_is_forgotten(run):
    run(FAILED_PLAN)


CAPTURE = r"""
text, _ = W.literal_set(seed=5, n_patterns=20, input_len=1000, plant_every=100)
ts = nb.TableSet([tables(text)])
data = np.zeros(1 << 20, np.uint8)
e = nb.Engine(0)


def batch(**kw):
    nb.batch_match_async(e, ts, data, [0, 1000], [1000, 500000], [0, 0], use_graph=True, result_capacity=CAP, **kw)


batch()
n = count("fake_instantiated")
batch()
assert count("fake_instantiated") == n  # replayed
keys = ctypes.c_void_p()
assert fake.cudaMalloc(ctypes.byref(keys), ctypes.c_size_t(64 * CAP)) == 0
held = e.memory()["reports"]
e.sort_unique_device(keys.value, 8 * CAP, keys.value)
assert e.memory()["reports"] > held  # the report buffers are others now
batch()
assert count("fake_instantiated") == n + 1  # captured again
batch()
assert count("fake_instantiated") == n + 1
batch(active_threshold=3)  # no kernel reads it
assert count("fake_instantiated") == n + 1
batch(unique=True)
assert count("fake_instantiated") == n + 2
"""


def test_capture_follows_the_buffers(run):
    run(CAPTURE)


SCRATCH = r"""
text, _ = W.literal_set(seed=5, n_patterns=200, input_len=1000, plant_every=100)
t = tables(text)
ts = nb.TableSet([t])
states = t.stats()["states"]
data = np.zeros(300_000, np.uint8)
SMS = 148
for queue in (0, 1024, 4096, 16384, 65536):
    e = nb.Engine(0)
    nb.batch_match_async(e, ts, data, [0], [len(data)], [0], result_capacity=CAP, queue_capacity=queue)
    slices = 2 * len(data) + 64 * (len(data) // 4 + 2 * len(data) // 249)  # candidates and runs
    # 16 warps with a worklist of the capacity and lists of every state
    per_warp = 4 * (max(queue or 65536, 1024) + 128 + states + states // 32 + 2)
    small = 32 if queue and queue < 16384 else 16  # small worklists are held whole by 32 warps
    assert e.memory()["scratch"] <= SMS * (16 * per_warp + 4 * (small - 16) * (queue + 128)) + slices
    if not 0 < queue < 16384:  # no more than 20 warps an SM took
        assert e.memory()["scratch"] - slices <= SMS * 20 * 4 * ((queue or 65536) + states + states // 32 + 2)
"""


def test_scratch_of_the_resident_warps(run):
    run(SCRATCH)


RESERVE = r"""
rng = np.random.default_rng(5)
dense = W.AnmlWriter("dense")  # most positions report: no filter
dense.ste("a", W.PRINTABLE[:60], ["b"], start="all-input", report=True)
dense.ste("b", W.PRINTABLE[:60], report=True)
loop = W.AnmlWriter("loop")    # cyclic
loop.ste("x", b"x", ["y"], start="all-input")
loop.ste("y", b"y", ["y", "z"])
loop.ste("z", b"z", report=True)
long = [bytes(rng.integers(97, 123, 8).astype(np.uint8)) for _ in range(3000)]
lists = W.AnmlWriter("lists")  # long lists in shallow tables: the shortest runs
for n, word in enumerate(long):
    for i, c in enumerate(word):
        lists.ste(f"r{n}_{i}", [ord("h") if i == 0 else c], [f"r{n}_{i + 1}"] if i < 7 else [],
                  start="all-input" if i == 0 else None, report=i == 7)
texts = [W.literal_set(seed=5, n_patterns=20, input_len=1000, plant_every=100)[0], dense.text(), loop.text(),
         W.dotstar_set(seed=6, n_patterns=40, input_len=1000, plant_every=100)[0], lists.text()]
ts = nb.TableSet([tables(t, depth=1, groups=3) for t in texts])
N = len(texts)
CHUNK, MOST, REQUESTS = 256, 3_000_001, 40
data = np.zeros(MOST, np.uint8)


def batch(e, lens, nfas, chunk):
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    nb.batch_match_async(e, ts, data[:int(sum(lens))], offs, lens, nfas, chunks=np.full(len(lens), chunk),
                         result_capacity=CAP, algorithm=algorithm)
    e.sync()


for algorithm in ("nonblockingpcgroups", "NAPgroups", "blockinggroups"):
    for lo, hi in ((CHUNK, 2048), (0, 0)):  # chunks chosen per request, or automatic
        e = nb.Engine(0)
        batch(e, [MOST], [0], lo)            # as a server warms up: one request, then the most
        each = MOST // REQUESTS
        batch(e, [each] * (REQUESTS - 1) + [MOST - each * (REQUESTS - 1)], np.arange(REQUESTS) % N, lo)
        held = e.memory()
        assert held["scratch"] > 0 and held["plan"] > 0
        for nfa in list(range(N)) + [-1] * 10:
            for size in (MOST, MOST // 7, 5000, 40):
                k = int(rng.integers(1, REQUESTS + 1)) if nfa < 0 else (1 if size == MOST // 7 else REQUESTS)
                cuts = np.sort(rng.integers(0, size + 1, k - 1))
                lens = np.diff(np.concatenate([[0], cuts, [size]]))
                nfas = rng.integers(0, N, k) if nfa < 0 else np.full(k, nfa)
                batch(e, lens, nfas, int(rng.integers(lo, hi + 1)))
                assert e.memory() == held, (algorithm, lo, nfa, size, k, held, e.memory())
"""


def test_batches_of_other_rules_allocate_nothing(run):
    run(RESERVE)


SORTS = r"""
# which sort a match ends with: the one-CTA kernel alone, or the graph with the pipeline
words, _ = W.literal_set(seed=5, n_patterns=6, input_len=1000, plant_every=100)
forks = W.AnmlWriter("forks")  # 2^9 paths to the end of a (b|b) c (b|b) c ...
for i in range(9):
    forks.ste(f"a{i}", b"a" if i == 0 else b"c", [f"b{i}", f"e{i}"], start="all-input" if i == 0 else None)
    for x in "be":
        forks.ste(f"{x}{i}", b"b", [f"a{i + 1}"])
forks.ste("a9", b"c", [], report=True)
loop = W.AnmlWriter("loop")
loop.ste("h", b"h", ["x", "y"], start="all-input")
for c in "xy":
    loop.ste(c, b"a", ["x", "y", "z"])
loop.ste("z", b"z", [], report=True)
t = [tables(x, depth=1) for x in (words, forks.text(), loop.text())]
ts = nb.TableSet(t)
data = np.zeros(4000, np.uint8)
e = nb.Engine(0)


def alone(f, *a, **kw):
    out = log(f, *a, **kw)
    graph, cta = any(x.startswith("graph") for x in out), any("sort_unique_cta" in x for x in out)
    assert graph != cta, out
    return cta


def plain(k, n):
    return alone(e.match_async, t[k], data, 1, n, result_capacity=CAP)


def batch(nfas, offs, lens):
    return alone(nb.batch_match_async, e, ts, data, offs, lens, nfas, result_capacity=CAP)


assert plain(0, 4000) and plain(0, 100)          # 4000 positions, 6 reports
assert plain(1, 4000) and plain(2, 4000)         # one report (however many paths lead to it)
big = np.zeros(70_000, np.uint8)
assert alone(e.match_async, t[1], big, 1, 65_536, result_capacity=CAP)
assert not alone(e.match_async, t[1], big, 1, 65_537, result_capacity=CAP)
assert batch([0, 0], [0, 2000], [2000, 2000])
assert not batch([0] * 30, [0] * 30, [4000] * 30)  # streams over the same bytes
assert batch([0] * 30, [0] * 30, [40] * 30)
assert batch([0, 1, 2], [0, 1000, 1100], [1000, 100, 0])


def captured(nfas, offs, lens):
    "In a capture nobody would finish a sort that left keys: the pipeline is there unless duplicates are bounded too."
    out = log(nb.batch_match_async, e, ts, data, offs, lens, nfas, result_capacity=CAP, use_graph=True)
    return not any("radix_scatter" in x for x in out)


assert captured([0, 0], [0, 2000], [2000, 2000])
assert captured([1], [0], [128]) and not captured([1], [0], [129])  # 512 paths to one report
assert not captured([2], [0], [1])                                  # cyclic: no bound
"""


def test_sorts_by_the_reports_that_can_come(run):
    run(SORTS)


KEEP = r"""
import weakref


class Tensor:  # a device tensor
    is_cuda = True

    def __init__(self, n):
        self.p = ctypes.c_void_p()
        assert fake.cudaMalloc(ctypes.byref(self.p), ctypes.c_size_t(n)) == 0
        self.n = n

    data_ptr = lambda self: self.p.value
    numel = lambda self: self.n
    element_size = lambda self: 1


text, _ = W.literal_set(seed=5, n_patterns=20, input_len=1000, plant_every=100)
t = tables(text)
ts = nb.TableSet([t])
e = nb.Engine(0)
for start in (lambda x: e.match_async(t, x, 1, 4096, result_capacity=CAP),
              lambda x: nb.batch_match_async(e, ts, x, [0], [4096], [0], result_capacity=CAP)):
    x = Tensor(4096)
    alive = weakref.ref(x)
    start(x)
    del x
    assert alive() is not None  # read in place: kept while the match runs
    e.sync()
    assert alive() is None      # and no longer
"""


def test_input_is_kept_until_the_match_has_ended(run):
    run(KEEP)
