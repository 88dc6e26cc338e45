"""Candidates whose lists are together many times a worklist: positions that
pass a look-ahead filter are those with the longest lists, and a run injects 32
of them at once. Every case gives the oracle's reports, with the smallest
worklists an engine takes and, for one large set, with the automatic ones."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu

LOWER = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz", np.uint8)
QUEUE = 1024  # entries beyond shared memory: the smallest capacity


def literals(words, start="all-input", writer=None, tag="w"):
    w = writer or W.AnmlWriter("words")
    for n, word in enumerate(words):
        for i, c in enumerate(word):
            w.ste(f"{tag}{n}_{i}", [c], [f"{tag}{n}_{i + 1}"] if i + 1 < len(word) else [],
                  start=start if i == 0 else None, report=i + 1 == len(word))
    return w


def tails(rng, n, lo, hi):
    return [bytes(rng.choice(LOWER, size=int(rng.integers(lo, hi + 1)))) for _ in range(n)]


def text_of(rng, words, size, between=b" "):
    """Words, whole and cut short, one after another."""
    out, at = [], 0
    while at < size:
        x = words[int(rng.integers(len(words)))]
        x = (x if rng.random() < 0.5 else x[:max(8, len(x) - int(rng.integers(1, 3)))]) + between
        out.append(x)
        at += len(x)
    return np.frombuffer(b"".join(out)[:size], np.uint8).copy()


def check(groups, data, queue, algorithm="nonblockingpcgroups", depth=-1, chunk=0):
    """One stream alone and beside another, through the batched entry."""
    tables = nb.Tables(groups, precompute_depth=depth)
    ts = nb.TableSet([tables])
    cut = len(data) // 3
    for offs, lens in (([0], [len(data)]), ([0, cut], [cut, len(data) - cut])):
        engine = nb.Engine(0)  # an engine keeps the largest queue it has held
        nb.batch_match_async(engine, ts, data, offs, lens, [0] * len(offs), algorithm=algorithm, chunk=chunk,
                             queue_capacity=queue)
        engine.sync()
        got = nb.split_by_stream(*nb.batch_results(engine), len(offs))
        wants = [oracle.match(groups.views(), data[o:o + n], 1, n)[0] for o, n in zip(offs, lens)]
        assert len(wants[0]) > 0
        for g, want in zip(got, wants):
            assert np.array_equal(g, want)


@pytest.mark.parametrize("rules", [40, 333, 1500])
@pytest.mark.parametrize("algorithm,depth", [("nonblockingpcgroups", -1), ("nonblockinggroups", 1),
                                             ("NAPgroups", 0)])
def test_shared_prefix(built, rules, algorithm, depth):
    rng = np.random.default_rng(rules)
    urls = [b"http://www." + t for t in tails(rng, rules, 4, 8)]
    groups = nb.Groups(nb.Nfa.from_string(literals(urls + tails(rng, 100, 6, 9)).text()), group_num=2)
    check(groups, text_of(rng, urls, 150_001), QUEUE, algorithm, depth)


@pytest.mark.parametrize("rules", [30, 31, 700])
def test_many_active_dotstar_rules(built, rules):
    """GET .*item<tail>: once all are active, each candidate tests every rule."""
    rng = np.random.default_rng(rules)
    ends = [b"item" + t for t in tails(rng, rules, 3, 6)]
    w = W.AnmlWriter("dotstar")
    for n, e in enumerate(ends):
        for i, c in enumerate(b"GET "):
            w.ste(f"g{n}_{i}", [c], [f"g{n}_{i + 1}"] if i < 3 else [f"s{n}", f"e{n}_0"],
                  start="all-input" if i == 0 else None)
        w.ste(f"s{n}", None, [f"s{n}", f"e{n}_0"], symbol_set="*")
        for i, c in enumerate(e):
            w.ste(f"e{n}_{i}", [c], [f"e{n}_{i + 1}"] if i + 1 < len(e) else [], report=i + 1 == len(e))
    groups = nb.Groups(nb.Nfa.from_string(w.text()), group_num=1)
    data = np.concatenate([np.frombuffer(b"GET ", np.uint8), text_of(rng, ends, 150_000)])
    check(groups, data, QUEUE)


@pytest.mark.parametrize("rules", [31, 33, 2500])
def test_many_start_of_data_rules(built, rules):
    rng = np.random.default_rng(rules)
    first = [b"header" + t for t in tails(rng, rules, 3, 6)]
    w = literals(first, start="start-of-data")
    groups = nb.Groups(nb.Nfa.from_string(literals(tails(rng, 80, 6, 9), writer=w, tag="x").text()), group_num=1)
    check(groups, np.concatenate([np.frombuffer(first[0], np.uint8), text_of(rng, first, 160_000)]), QUEUE)


def test_shared_prefix_with_automatic_worklists(engine):
    """3000 rules of one prefix, as long as the tables are deep, beside 500 others
    (the mean list is short), on 150 KB of ten-byte names: one injection is 75,000 entries, more than the automatic
    worklist holds."""
    rng = np.random.default_rng(9)
    names = [b"http:/" + t for t in tails(rng, 3000, 3, 3)]
    groups = nb.Groups(nb.Nfa.from_string(literals(names + tails(rng, 500, 6, 9)).text()), group_num=1)
    data = np.frombuffer(b"".join(names[i] + b" " for i in rng.integers(0, 3000, 15_000)), np.uint8)
    want, _ = oracle.match(groups.views(), data, 1, len(data))
    for _ in range(2):
        got = engine.match(nb.Tables(groups, precompute_depth=-1), data, 1, len(data))
        assert len(want) >= 15_000 and np.array_equal(got, want)


def side_paths(rules, length):
    """h a a a ...: every symbol matches the next state and three that end there."""
    w = W.AnmlWriter("side")
    for n in range(rules):
        for i in range(length):
            w.ste(f"p{n}_{i}", b"h" if i == 0 else b"a", [f"p{n}_{i + 1}"] + [f"d{n}_{i}_{k}" for k in range(3)]
                  if i + 1 < length else [], start="all-input" if i == 0 else None, report=i + 1 == length)
        for i in range(3 * length - 3):
            w.ste(f"d{n}_{i // 3}_{i % 3}", b"a", [])
    return nb.Groups(nb.Nfa.from_string(w.text()), group_num=1)


@pytest.mark.parametrize("size", [20_000, 160_000])  # looked up position by position, and scanned
@pytest.mark.parametrize("length", [60, 400, 2047])
@pytest.mark.parametrize("algorithm", ["nonblockingallgroups", "NAPgroups"])
def test_side_paths(built, size, length, algorithm):
    """Long paths that leave three short ones at every symbol: 32 of them
    followed side by side leave 96 entries a symbol, which wait for the paths' end."""
    groups = side_paths(40 if length < 1000 else 10, length)
    data = np.resize(np.frombuffer(b"h" + b"a" * (length - 1 if length > 1000 else length + 5), np.uint8), size)
    check(groups, data, QUEUE, algorithm)


def test_side_paths_with_automatic_worklists(engine):
    groups = side_paths(40, 1400)
    tables = nb.Tables(groups, precompute_depth=-1)
    for size in (30_000, 160_000):
        data = np.resize(np.frombuffer(b"h" + b"a" * 1500, np.uint8), size)
        want, _ = oracle.match(groups.views(), data, 1, len(data))
        assert len(want) > 0 and np.array_equal(engine.match(tables, data, 1, len(data)), want)
