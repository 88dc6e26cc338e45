"""Look-ahead filters: a position whose bit is clear must need no injection.

CPU: a C++ program plans the tiles and filters of an automaton, then walks
random and accepted class strings through the tile's graph from the states it
injects: a path that is alive after `len` symbols, or a report within them,
needs its bit set, and no report may come before `min_rep` symbols.
GPU: matches against the oracle at sizes around the filter's lengths, scan
steps, pieces and segment ends.
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
#include <cstdlib>
#include <random>
#include <set>
#include "handles.h"
#include "tables.h"
using namespace ngap;
int main(int argc, char** argv) {
  ngap_nfa* n = nullptr;
  ngap_groups* g = nullptr;
  if (argc != 5 || ngap_nfa_load_anml(argv[1], &n) != NGAP_OK) return 2;
  ngap_group_opts go{atoi(argv[2]), -1, 1, 0};
  if (ngap_groups_build(n, &go, &g) != NGAP_OK) return 3;
  TableOpts to;
  to.precompute_depth = 1;
  to.tile_mode = atoi(argv[3]);
  std::vector<TileHost> tiles;
  if (build_tiles(g->gs, to, tiles) != NGAP_OK) return 4;
  build_filters(tiles);
  std::mt19937 rng(atoi(argv[4]));
  int nf = 0;
  long clear = 0, total = 0;
  for (const TileHost& t : tiles) {
    const FilterHost& f = t.filt;
    if (f.len == 0) continue;
    nf++;
    auto ok = [&](uint32_t v, int c) { return (t.cmask[(size_t)v * t.cw + (c >> 5)] >> (c & 31)) & 1u; };
    auto rep = [&](uint32_t v) { return (t.rep[v >> 5] >> (v & 31)) & 1u; };
    std::set<uint32_t> src(t.aas.begin(), t.aas.end());
    if (t.phase == 2)
      for (uint32_t a : t.act_local)
        for (int j = 0; j < 4; j++) {
          const uint32_t u = t.succ[(size_t)(a & kActIdMask) * 4 + j];
          if (u != kNoSucc) src.insert(u & 0x7fffffffu);
        }
    const std::vector<uint32_t> from(src.begin(), src.end());
    for (int it = 0; it < 4000; it++) {
      std::vector<int> s(f.len);
      for (int& c : s) c = rng() % t.ncls;
      if (it & 1) {  // follow a path from a source, then perhaps change a symbol
        uint32_t v = from[rng() % from.size()];
        for (int i = 0; i < f.len; i++) {
          std::vector<int> acc;
          for (int c = 0; c < t.nlive; c++)
            if (ok(v, c)) acc.push_back(c);
          if (acc.empty()) break;
          s[i] = acc[rng() % acc.size()];
          std::vector<uint32_t> nx;
          for (int k = 0; k < 4; k++)
            if (t.succ[(size_t)v * 4 + k] != kNoSucc) nx.push_back(t.succ[(size_t)v * 4 + k] & 0x7fffffffu);
          if (nx.empty()) break;
          v = nx[rng() % nx.size()];
        }
        if (it & 2) s[rng() % f.len] = rng() % t.ncls;
      }
      std::set<uint32_t> cur;
      for (uint32_t v : from)
        if (ok(v, s[0])) cur.insert(v);
      bool need = false;
      for (int d = 1; d <= f.len; d++) {
        for (uint32_t v : cur)
          if (rep(v)) {
            if (d < f.min_rep) return printf("report after %d symbols, min_rep %d\n", d, f.min_rep), 1;
            need = true;
          }
        if (d == f.len) break;
        std::set<uint32_t> nx;
        for (uint32_t v : cur)
          for (int k = 0; k < 4; k++) {
            const uint32_t u = t.succ[(size_t)v * 4 + k];
            if (u != kNoSucc && ok(u & 0x7fffffffu, s[d])) nx.insert(u & 0x7fffffffu);
          }
        cur.swap(nx);
      }
      need = need || !cur.empty();
      uint32_t h = 0;
      for (int c : s) h = h * kFilterMul + (uint32_t)c;
      const uint64_t m = filter_mask(h);
      const bool set = (f.blocks[(h * kFilterBlock) >> f.shift] & m) == m;
      if (need && !set) return printf("tile phase %d: a needed position is filtered out\n", t.phase), 1;
      if (!(it & 1)) {
        total++;
        clear += !set;
      }
    }
  }
  printf("ok filters %d tiles %d clear %.3f\n", nf, (int)tiles.size(), total ? (double)clear / total : 1.0);
  ngap_groups_destroy(g);
  ngap_nfa_destroy(n);
  return 0;
}
"""


@pytest.fixture(scope="module")
def checker(built, tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(cuda, "include", "vector_types.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("filter")
    (d / "check.cpp").write_text(CHECK)
    lib = os.path.join(ROOT, "ngap_b200")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(lib, "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"),
                    str(d / "check.cpp"), "-o", str(d / "check"), "-L", lib, "-lngap_b200",
                    "-Wl,-rpath," + lib], check=True, capture_output=True, text=True)
    return str(d / "check")


def short_rules(rng, n, lo, hi, alpha):
    """Literals of lo..hi symbols over alpha, with a few classes."""
    w = W.AnmlWriter("short")
    for p in range(n):
        L = int(rng.integers(lo, hi + 1))
        for i in range(L):
            cls = set(rng.choice(alpha, size=1 + 2 * int(rng.random() < 0.2)).tolist())
            w.ste(f"p{p}_{i}", cls, targets=[f"p{p}_{i + 1}"] if i + 1 < L else [],
                  start="all-input" if i == 0 else None, report=(i == L - 1))
    return w.text()


BYTES = np.arange(20, 220, dtype=np.uint8)
BYTES_LAW = np.arange(1, 201) ** -1.3 / np.sum(np.arange(1, 201) ** -1.3)


def wide_dotstar(rng, n):
    """a{2,4} .* b{2,5} over a large alphabet (more than three class words)."""
    w = W.AnmlWriter("wide")
    for p in range(n):
        a, b = int(rng.integers(2, 5)), int(rng.integers(2, 6))
        for i in range(a):
            w.ste(f"w{p}a{i}", [int(rng.choice(BYTES, p=BYTES_LAW))],
                  [f"w{p}a{i + 1}"] if i + 1 < a else [f"w{p}s", f"w{p}b0"],
                  start="all-input" if i == 0 else None)
        w.ste(f"w{p}s", None, [f"w{p}s", f"w{p}b0"], symbol_set="*")
        for i in range(b):
            w.ste(f"w{p}b{i}", [int(rng.choice(BYTES, p=BYTES_LAW))], [f"w{p}b{i + 1}"] if i + 1 < b else [],
                  report=(i == b - 1))
    return w.text()


def mixed_alphabets(seed):
    """Edit-distance rules over ACGT beside dot-star rules over text: (ANML, input)."""
    w, rng = W.AnmlWriter("mix"), np.random.default_rng(seed)
    _, dna = W.levenshtein_set(n_patterns=12, input_len=80_000, plant_every=997, writer=w, rng=rng)
    _, text = W.dotstar_set(n_patterns=60, input_len=85_000, plant_every=997, writer=w, rng=rng)
    return w.text(), np.concatenate([dna, text])


def rule_sets():
    rng = np.random.default_rng(31)
    kw = dict(input_len=1 << 12, plant_every=1 << 8)
    return {
        "hamming": W.hamming_set(seed=3, n_patterns=30, **kw)[0],
        "motif": W.hamming_set(seed=4, n_patterns=40, k=8, d=1, **kw)[0],
        "levenshtein": W.levenshtein_set(seed=5, n_patterns=12, **kw)[0],
        "dotstar": W.dotstar_set(seed=6, n_patterns=60, **kw)[0],
        "literal": W.literal_set(seed=7, n_patterns=40, **kw)[0],
        "short": short_rules(rng, 12, 2, 9, W.PRINTABLE),
        "dense": short_rules(rng, 30, 1, 4, W.PRINTABLE[:20]),
        "one": short_rules(rng, 3, 1, 1, W.PRINTABLE),
        "mix": mixed_alphabets(33)[0],
        "wide": wide_dotstar(np.random.default_rng(32), 400),
        "mixed": short_rules(rng, 60, 3, 20, W.PRINTABLE[:20]),
    }


@pytest.mark.parametrize("name", list(rule_sets()))
@pytest.mark.parametrize("groups,mode", [(1, 0), (3, 1), (3, 2)])
def test_filter_covers_every_path(checker, tmp_path, name, groups, mode):
    anml = tmp_path / "rules.anml"
    anml.write_text(rule_sets()[name])
    r = subprocess.run([checker, str(anml), str(groups), str(mode), "9"], capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    filters, clear = int(r.stdout.split()[2]), float(r.stdout.split()[6])
    if name not in ("one", "dense"):
        assert filters > 0 and clear > 0.5, r.stdout


@pytest.mark.parametrize("groups,mode", [(1, "shared"), (1, "auto")])
def test_small_alphabets_get_their_own_tiles(built, groups, mode):
    both = nb.Groups(nb.Nfa.from_string(mixed_alphabets(33)[0]), group_num=groups)
    lev = W.levenshtein_set(n_patterns=12, input_len=1 << 12, plant_every=1 << 8)[0]
    states = sum(t["num_states"] for t in nb.Groups(nb.Nfa.from_string(lev), group_num=groups).tiles())
    tiles = both.tiles(tile_mode=mode)
    dna = [t for t in tiles if t["phase"] == 0 and t["nlive"] == 4]
    assert len(dna) == groups and sum(t["num_states"] for t in dna) == states
    assert all(t["nlive"] > 8 for t in tiles if t not in dna)
    # one alphabet alone stays one tile per group
    alone = nb.Groups(nb.Nfa.from_string(lev), group_num=1).tiles(tile_mode="shared")
    assert len(alone) == 1


# inputs of 128 Ki positions and more are scanned, shorter ones looked up position
# by position (unless their tables' lists are long)
LENGTH = 165_000


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["hamming", "motif", "dotstar", "dense", "mixed", "mix", "wide"])
def test_filtered_matches(engine, name):
    anml = rule_sets()[name]
    groups = nb.Groups(nb.Nfa.from_string(anml), group_num=2)
    rng = np.random.default_rng(17)
    alpha = W.ACGT if name in ("hamming", "motif") else W.PRINTABLE
    gen = {"hamming": lambda: W.hamming_set(seed=3, n_patterns=30, input_len=LENGTH, plant_every=97)[1],
           "motif": lambda: W.hamming_set(seed=4, n_patterns=40, k=8, d=1, input_len=LENGTH,
                                          plant_every=61)[1],
           "mix": lambda: mixed_alphabets(33)[1],
           "dotstar": lambda: W.dotstar_set(seed=6, n_patterns=60, input_len=LENGTH, plant_every=97)[1]}
    data = gen[name]() if name in gen else rng.choice(W.PRINTABLE[:20], size=LENGTH).astype(np.uint8)
    if name == "wide":
        data = rng.choice(BYTES, size=LENGTH, p=BYTES_LAW).astype(np.uint8)
    data = data.copy()
    data[rng.integers(0, len(data), 800)] = rng.choice(alpha, size=800)
    data[1000:1040] = 0  # bytes no state accepts
    some = 0
    for mode, depth in (("shared", 1), ("shared", 3), ("global", -1)):
        tables = nb.Tables(groups, precompute_depth=depth, tile_mode=mode)
        for num_seg, seg_len in ((1, 1), (3, 15), (1, 257), (2, 2065), (5003, 31), (1201, 113), (517, 257),
                                 (38, 4099), (1, 163_841)):
            for algo, chunk, window in (("nonblockingpcgroups", 0, 0), ("nonblockingallgroups", 33, 64),
                                        ("NAPgroups", 300, 0), ("nonblockinggroups", 0, 100)):
                got = engine.match(tables, data[:num_seg * seg_len], num_seg, seg_len, algorithm=algo,
                                   chunk=chunk, window=window)
                want, _ = oracle.match(groups.views(), data[:num_seg * seg_len], num_seg, seg_len)
                some += len(want)
                assert np.array_equal(got, want), (mode, depth, num_seg, seg_len, algo)
    assert some > 0
