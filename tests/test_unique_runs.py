"""--unique on tiles that are scanned: paths that meet are followed once."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


def diamonds(n, dotstar):
    """a (b|b) c (b|b) c ... : two states for every b, so 2^n paths to the end; a
    .* in front of it where dotstar is set."""
    w = W.AnmlWriter("diamonds")
    if dotstar:
        w.ste("g", b"G", ["s", "a0"], start="all-input")
        w.ste("s", None, ["s", "a0"], symbol_set="*")
    for i in range(n):
        w.ste(f"a{i}", b"a" if i == 0 else b"c", [f"b{i}", f"e{i}"],
              start="all-input" if i == 0 and not dotstar else None)
        for x in "be":
            w.ste(f"{x}{i}", b"b", [f"a{i + 1}"])
    w.ste(f"a{n}", b"c", [], report=True)
    return nb.Groups(nb.Nfa.from_string(w.text()), group_num=1)


@pytest.mark.parametrize("size", [30_001, 200_001])  # looked up position by position, and scanned
@pytest.mark.parametrize("dotstar", [False, True])
@pytest.mark.parametrize("n", [1, 6, 9])
def test_paths_that_meet(engine, size, dotstar, n):
    groups = diamonds(n, dotstar)
    data = np.random.default_rng(size).choice(np.frombuffer(b"xyzwvuts", np.uint8), size=size).astype(np.uint8)
    data[0] = ord("G")
    word = np.frombuffer(b"a" + b"bc" * n, np.uint8)
    for at in range(100, size - 50, 4999):
        data[at:at + len(word)] = word
    data[-len(word) - 3:-3] = word
    want, _ = oracle.match(groups.views(), data, 1, size)
    assert len(want) > 0
    tables = nb.Tables(groups, precompute_depth=1)
    raw = {}
    for unique in (False, True):
        got = engine.match(tables, data, 1, size, unique=unique)
        assert np.array_equal(got, want)
        raw[unique] = engine.counts()[0]
        nb.batch_match_async(engine, nb.TableSet([tables]), data, [0, 0], [size, size // 2], [0, 0], unique=unique)
        engine.sync()
        rep, sid = nb.batch_results(engine)
        assert np.array_equal(rep[sid == 0], want)
        assert np.array_equal(rep[sid == 1], want[(want & np.uint64(0xFFFFFFFF)) < size // 2])
    assert raw[False] == len(want) << n  # every path reports
    # the planted words are apart: one path to the last b, and both of its states report
    assert raw[True] == 2 * len(want)


def test_meeting_paths_stay_within_the_result_capacity(engine):
    groups = diamonds(12, False)
    data = np.full(200_000, ord("x"), np.uint8)
    word = np.frombuffer(b"a" + b"bc" * 12, np.uint8)
    for at in range(0, 200_000 - 50, 1000):
        data[at:at + len(word)] = word
    want, _ = oracle.match(groups.views(), data, 1, len(data))
    tables = nb.Tables(groups, precompute_depth=1)
    got = engine.match(tables, data, 1, len(data), unique=True, result_capacity=2 * len(want))
    assert np.array_equal(got, want)
