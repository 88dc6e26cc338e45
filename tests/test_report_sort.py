"""Report compaction at the edges of its ranges: the bitonic, shared-memory and
global passes of the one-CTA sort and the radix pipeline, chosen by the number
of reports and the length of the input."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rules():
    w = W.AnmlWriter("bytes")
    for i, c in enumerate(b"abc"):  # a report per byte, two for 'c'
        w.ste(f"r{i}", [c], start="all-input", report=True)
    w.ste("again", [ord("c")], start="all-input", report=True)
    groups = nb.Groups(nb.Nfa.from_string(w.text()), group_num=3)
    return nb.Tables(groups, precompute_depth=1)


@pytest.fixture(scope="module")
def one(rules):
    return nb.TableSet([rules])


def expected(tables, data):
    """(id, offset) pairs by byte, in the reference's order."""
    views = tables.groups.views()
    out = []
    for g, v in enumerate(views):
        for s in range(v.num_states):
            syms = [b for b in range(256) if (int(v.symbol_sets[s, b >> 5]) >> (b & 31)) & 1]
            at = np.flatnonzero(np.isin(data, syms)).astype(np.uint64)
            out.append((np.uint64(s | g << 22) << np.uint64(32)) | at)
    r = np.concatenate(out)
    return r[np.lexsort((r >> np.uint64(32), r & np.uint64(0xFFFFFFFF)))]


@pytest.mark.parametrize("length", [16_000, 300_001])  # one CTA alone, or with the pipeline
@pytest.mark.parametrize("hits", [0, 1, 31, 512, 1023, 1024, 1025, 4097, 8190, 8192, 8194, 70_000])
def test_match_reports(engine, rules, one, length, hits):
    hits = min(hits, length)
    rng = np.random.default_rng(hits + length)
    data = np.full(length, ord("x"), np.uint8)
    at = rng.choice(length, size=hits, replace=False)
    data[at] = rng.choice(np.frombuffer(b"ab", np.uint8), size=hits)
    if hits > 2:
        data[at[0]] = ord("c")  # two reports
    want = expected(rules, data)
    assert len(want) == hits + (hits > 2)
    for _ in range(2):  # the second match starts from what the first left behind
        got = engine.match(rules, data, 1, length)
        assert np.array_equal(got, want)
        assert engine.counts()[1] == len(want)
    lens = np.array([length // 3, length - length // 3, 0])
    offs = np.array([0, length // 3, length])
    for use_graph in (False, True):
        if use_graph:
            import torch
            inp = torch.from_numpy(data).cuda()
        else:
            inp = data
        nb.batch_match_async(engine, one, inp, offs, lens, [0, 0, 0], use_graph=use_graph)
        engine.sync()
        rep, sid = nb.batch_results(engine)
        parts = nb.split_by_stream(rep, sid, 3)
        for k in range(3):
            assert np.array_equal(parts[k], expected(rules, data[offs[k]:offs[k] + lens[k]]))
    engine.match_async(rules, data, 1, length, report_off=True)
    engine.sync()
    assert engine.counts() == (len(want), 0)


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 2047, 2049, 8191, 8192, 8193, 262_147])
@pytest.mark.parametrize("spread", ["wide", "narrow", "equal"])
def test_sort_unique_device(engine, n, spread):
    import torch
    rng = np.random.default_rng(n)
    hi = {"wide": 1 << 32, "narrow": 40, "equal": 1}[spread]
    keys = (rng.integers(0, hi, n, dtype=np.uint64) << np.uint64(32)) | rng.integers(
        0, hi, n, dtype=np.uint64)
    d_in = torch.from_numpy(keys.view(np.int64)).cuda()
    d_out = torch.empty_like(d_in)
    m = engine.sort_unique_device(d_in.data_ptr(), n, d_out.data_ptr())
    s = np.unique((keys << np.uint64(32)) | (keys >> np.uint64(32)))
    want = (s << np.uint64(32)) | (s >> np.uint64(32))
    assert m == len(want)
    assert np.array_equal(d_out[:m].cpu().numpy().view(np.uint64), want)
