"""Which rules get a tile of their own for their small alphabet: a large share
over one alphabet beside others, never the many small alphabets of short words
(every tile is one more scan of the input)."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W

LOWER = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz", np.uint8)
DIGITS = np.frombuffer(b"01234567", np.uint8)


def words(seed, n, lo, hi, alpha=LOWER):
    rng = np.random.default_rng(seed)
    return [rng.choice(alpha, size=int(rng.integers(lo, hi + 1))).tolist() for _ in range(n)]


def tiles(rules, groups, mode):
    w = W.AnmlWriter("words")
    for n, word in enumerate(rules):
        for i, c in enumerate(word):
            w.ste(f"w{n}_{i}", [c], [f"w{n}_{i + 1}"] if i + 1 < len(word) else [],
                  start="all-input" if i == 0 else None, report=i + 1 == len(word))
    g = nb.Groups(nb.Nfa.from_string(w.text()), group_num=groups)
    return g.tiles(precompute_depth=2, tile_mode=mode)


@pytest.mark.parametrize("groups,mode,want", [(1, "auto", 1), (1, "global", 1), (10, "auto", 1), (10, "shared", 10)])
def test_short_words_share_a_tile(built, groups, mode, want):
    rules = [list(b"http:/") + t for t in words(1, 2000, 3, 3)] + words(2, 6000, 3, 9)
    assert len(tiles(rules, groups, mode)) == want


@pytest.mark.parametrize("groups,mode", [(1, "auto"), (1, "shared"), (10, "auto"), (10, "shared")])
def test_one_small_alphabet_and_its_subsets_share_a_tile(built, groups, mode):
    # short strings over four bases: many use two or three of them
    assert len(tiles(words(3, 400, 3, 8, W.ACGT), groups, mode)) == groups


@pytest.mark.parametrize("mode", ["auto", "shared"])
def test_a_large_share_gets_its_own_tile(built, mode):
    text = words(4, 300, 9, 16)
    for dna, apart in ((200, True), (100, True), (10, False)):
        t = tiles(words(5, dna, 4, 12, W.ACGT) + text, 1, mode)
        own = [x for x in t if x["nlive"] == 4]
        # its own tile, with the rules that use fewer bases; too few rules: none
        assert len(t) == 1 + apart and len(own) == apart
        assert not apart or own[0]["num_ccs"] == dna
    t = tiles(words(6, 200, 8, 12, W.ACGT) + words(7, 200, 8, 12, DIGITS) + text, 1, mode)
    assert sorted(x["nlive"] for x in t)[:2] == [4, 8] and len(t) == 3
