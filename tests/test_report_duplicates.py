"""Short inputs whose reports are few but emitted once for each of very many
paths: more keys than the one-CTA sort takes are left to the pipeline, which the
sync launches, and nothing of it shows in the next match."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case(built):
    w = W.AnmlWriter("forks")  # a (b|b) c (b|b) c ...: 2^12 paths
    n = 12
    for i in range(n):
        w.ste(f"a{i}", b"a" if i == 0 else b"c", [f"b{i}", f"e{i}"], start="all-input" if i == 0 else None)
        for x in "be":
            w.ste(f"{x}{i}", b"b", [f"a{i + 1}"])
    w.ste(f"a{n}", b"c", [], report=True)
    groups = nb.Groups(nb.Nfa.from_string(w.text()), group_num=1)
    return groups, nb.Tables(groups, precompute_depth=1), b"a" + b"bc" * n


# words of 4096 reports each: below 8192, below and above 65,536, several times that
@pytest.mark.parametrize("words", [0, 1, 3, 15, 17, 90])
def test_many_duplicates(built, case, words):
    groups, tables, word = case
    data = np.full(6000, ord("x"), np.uint8)
    for k in range(words):
        data[k * 60 + 7:k * 60 + 7 + len(word)] = np.frombuffer(word, np.uint8)
    want, _ = oracle.match(groups.views(), data, 1, len(data))
    assert len(want) == words
    clean = np.full(6000, ord("x"), np.uint8)
    engine, ts = nb.Engine(0), nb.TableSet([tables])
    for _ in range(2):
        got = engine.match(tables, data, 1, len(data))
        assert np.array_equal(got, want) and engine.counts() == (words << 12, words)
        engine.sync()  # once more: nothing left to do
        assert engine.counts() == (words << 12, words)
        assert engine.match(tables, clean, 1, len(clean)).size == 0 and engine.counts() == (0, 0)
    # a match that nobody waited for, then another
    engine.match_async(tables, data, 1, len(data))
    assert engine.match(tables, clean, 1, len(clean)).size == 0 and engine.counts() == (0, 0)
    engine.match_async(tables, data, 1, len(data))
    assert np.array_equal(engine.match(tables, data, 1, len(data)), want)
    # batched, plain and captured
    for use_graph in (False, True, True):
        import torch
        src = torch.from_numpy(data).cuda()
        nb.batch_match_async(engine, ts, src, [0, 0, 3000], [6000, 0, 3000], [0, 0, 0], use_graph=use_graph)
        engine.sync()
        a, _, c = nb.split_by_stream(*nb.batch_results(engine), 3)
        assert np.array_equal(a, want)
        assert np.array_equal(c, oracle.match(groups.views(), data[3000:], 1, 3000)[0])
    # a standalone sort between the match and its sync
    import torch
    keys = torch.from_numpy(np.random.default_rng(words).integers(0, 1 << 40, 300_000)).cuda()
    out = torch.empty_like(keys)
    engine.match_async(tables, data, 1, len(data), result_capacity=1 << 20)
    n = engine.sort_unique_device(keys.data_ptr(), len(keys), out.data_ptr())
    engine.sync()
    assert n == len(torch.unique(keys)) and np.array_equal(engine.results(), want)
