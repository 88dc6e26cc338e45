"""The blocking algorithm looks at a state once a position: whole windows where
few paths can meet in a state, windows of one position elsewhere.

CPU: the bound on meeting paths against every input of small automata. GPU:
cyclic and forked rules whose paths no kernel could follow one by one."""
import itertools
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
#include <cstdlib>
#include "handles.h"
#include "tables.h"
using namespace ngap;
// the rule file's tiles: bound on the paths that meet, and on those that report
int main(int argc, char** argv) {
  ngap_nfa* n = nullptr;
  ngap_groups* g = nullptr;
  if (argc != 2 || ngap_nfa_load_anml(argv[1], &n) != NGAP_OK) return 2;
  ngap_group_opts go{1, -1, 1, 0};
  if (ngap_groups_build(n, &go, &g) != NGAP_OK) return 3;
  TableOpts to;
  to.precompute_depth = 1;
  std::vector<TileHost> tiles;
  if (build_tiles(g->gs, to, tiles) != NGAP_OK) return 4;
  for (TileHost& t : tiles) {
    count_paths(t);
    printf("%d %g %g %d\n", t.phase, t.max_paths, t.report_paths, many_paths(t.max_paths));
  }
  ngap_groups_destroy(g);
  ngap_nfa_destroy(n);
  return 0;
}
"""


@pytest.fixture(scope="module")
def bounds(built, tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(cuda, "include", "vector_types.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("paths")
    (d / "check.cpp").write_text(CHECK)
    lib = os.path.join(ROOT, "ngap_b200")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(lib, "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"),
                    str(d / "check.cpp"), "-o", str(d / "check"), "-L", lib, "-lngap_b200",
                    "-Wl,-rpath," + lib], check=True, capture_output=True, text=True)

    def of(anml):
        (d / "rules.anml").write_text(anml)
        out = subprocess.run([str(d / "check"), str(d / "rules.anml")], check=True, capture_output=True, text=True)
        return [tuple(float(x) for x in line.split()) for line in out.stdout.splitlines()]
    return of


def forks(n):
    """a (b|b) c (b|b) c ...: 2^n paths to the end."""
    w = W.AnmlWriter("forks")
    for i in range(n):
        w.ste(f"a{i}", b"a" if i == 0 else b"c", [f"b{i}", f"e{i}"], start="all-input" if i == 0 else None)
        for x in "be":
            w.ste(f"{x}{i}", b"b", [f"a{i + 1}"])
    w.ste(f"a{n}", b"c", [], report=True)
    return w.text()


def loops():
    """h (a|a)+ z: two states that follow each other and themselves."""
    w = W.AnmlWriter("loops")
    w.ste("h", b"h", ["x", "y"], start="all-input")
    for s in "xy":
        w.ste(s, b"a", ["x", "y", "z"])
    w.ste("z", b"z", [], report=True)
    return w.text()


def random_acyclic(seed):
    """(ANML, states): up to eight states over three symbols, edges forward only, in one component."""
    rng = np.random.default_rng(seed)
    n = int(rng.integers(3, 9))
    states = []
    for v in range(n):
        later = [u for u in range(v + 1, n) if rng.random() < 0.5][:4]
        if v + 1 < n and not later:
            later = [v + 1]
        syms = [s for s in range(3) if rng.random() < 0.6] or [int(rng.integers(3))]
        states.append((syms, later, v == 0 or rng.random() < 0.2, v == n - 1 or rng.random() < 0.3))
    w = W.AnmlWriter("random")
    for v, (syms, later, start, rep) in enumerate(states):
        w.ste(f"s{v}", [97 + s for s in syms], [f"s{u}" for u in later], start="all-input" if start else None,
              report=rep)
    return w.text(), states


@pytest.mark.parametrize("seed", range(25))
def test_bound_covers_every_input(bounds, seed):
    anml, states = random_acyclic(seed)
    got = bounds(anml)
    most = reports = 0
    n = len(states)
    for s in itertools.product(range(3), repeat=min(n, 6)):
        paths = [0] * n  # that end in each state at the current position
        for c in s:
            now = [0] * n
            for v, (syms, _, start, _) in enumerate(states):
                if c in syms:
                    into = sum(paths[u] for u in range(n) if v in states[u][1])
                    now[v] = 1 if start else into  # edges into always-active states are dropped
            paths = now
            most = max(most, max(paths))
            reports = max(reports, sum(p for p, x in zip(paths, states) if x[3]))
    assert most <= max(t[1] for t in got) and reports <= sum(t[2] for t in got)


def test_bound_of_known_rules(bounds):
    kw = dict(input_len=1 << 12, plant_every=1 << 8)
    for anml in (W.literal_set(seed=7, n_patterns=40, **kw)[0], W.hamming_set(seed=3, n_patterns=30, **kw)[0]):
        assert all(t[1] == 1 and not t[3] for t in bounds(anml))
    assert [t[1:] for t in bounds(forks(3))] == [(8.0, 8.0, 0.0)]
    assert [t[1:] for t in bounds(forks(10))] == [(1024.0, 1024.0, 0.0)]
    assert [t[1:] for t in bounds(forks(11))] == [(2048.0, 2048.0, 1.0)]
    assert [t[1:] for t in bounds(loops())] == [(np.inf, np.inf, 1.0)]
    # followed in whole windows: the dot-star pairs, and edit distance
    assert not any(t[3] for t in bounds(W.dotstar_set(seed=6, n_patterns=60, **kw)[0]))
    assert not any(t[3] for t in bounds(W.levenshtein_set(seed=5, n_patterns=12, **kw)[0]))


@pytest.mark.gpu
@pytest.mark.parametrize("size", [5_000, 200_000])
@pytest.mark.parametrize("rules", ["loops", "forks"])
def test_blocking_follows_states(engine, size, rules):
    groups = nb.Groups(nb.Nfa.from_string(loops() if rules == "loops" else forks(40)), group_num=1)
    word = b"h" + b"a" * 200 + b"z" if rules == "loops" else b"a" + b"bc" * 40 + b"xy"
    data = np.resize(np.frombuffer(word, np.uint8), size)
    want, _ = oracle.match(groups.views(), data, 1, size)
    assert len(want) > 0
    tables = nb.Tables(groups, precompute_depth=1)
    assert np.array_equal(engine.match(tables, data, 1, size, algorithm="blockinggroups"), want)
    assert engine.counts()[0] == 2 * len(want)  # from each of the two states before
    nb.batch_match_async(engine, nb.TableSet([tables]), data, [0], [size], [0], algorithm="blockinggroups")
    engine.sync()
    assert np.array_equal(nb.batch_results(engine)[0], want)


@pytest.mark.gpu
@pytest.mark.parametrize("size", [5_000, 200_000])
def test_blocking_reports_few_duplicates(engine, size):
    """Forks followed in whole windows: 2^8 paths, two states before the report."""
    groups = nb.Groups(nb.Nfa.from_string(forks(8)), group_num=1)
    data = np.full(size, ord("x"), np.uint8)
    word = np.frombuffer(b"a" + b"bc" * 8, np.uint8)
    for at in range(50, size - 50, 997):
        data[at:at + len(word)] = word
    want, _ = oracle.match(groups.views(), data, 1, size)
    tables = nb.Tables(groups, precompute_depth=1)
    cap = 2 * len(want)
    assert np.array_equal(engine.match(tables, data, 1, size, algorithm="blockinggroups", result_capacity=cap), want)
    nb.batch_match_async(engine, nb.TableSet([tables]), data, [0], [size], [0], algorithm="blockinggroups",
                         result_capacity=cap)
    engine.sync()
    assert np.array_equal(nb.batch_results(engine)[0], want)


@pytest.mark.gpu
@pytest.mark.parametrize("algorithm", ["blockinggroups", "NAPgroups"])
@pytest.mark.parametrize("size", [3_000, 150_000])
def test_many_always_active_states_of_one_symbol(built, algorithm, size):
    """1200 rules that start with the same byte, 32 of it in a row, and the
    smallest worklists."""
    rng = np.random.default_rng(size)
    w = W.AnmlWriter("same")
    for n in range(1290):
        first = ord("h") if n < 1200 else 33 + (n - 1200) % 60
        w.ste(f"r{n}", [first], [f"s{n}"], start="all-input")
        w.ste(f"s{n}", [int(rng.integers(33, 120))], [], report=True)
    groups = nb.Groups(nb.Nfa.from_string(w.text()), group_num=1)
    data = rng.integers(33, 120, size).astype(np.uint8)
    data[500:700] = ord("h")
    want, _ = oracle.match(groups.views(), data, 1, size)
    engine = nb.Engine(0)
    nb.batch_match_async(engine, nb.TableSet([nb.Tables(groups, precompute_depth=1)]), data, [0], [size], [0],
                         algorithm=algorithm, queue_capacity=1024)
    engine.sync()
    assert len(want) > 0 and np.array_equal(nb.batch_results(engine)[0], want)
