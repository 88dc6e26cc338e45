"""A captured batch after its engine's device buffers have moved: the next call
with the same arguments captures again instead of replaying old addresses."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu

CAP = 8192  # report capacity of the batch


@pytest.mark.parametrize("grow", ["sort", "capacity", "streams", "plain"])
def test_graph_after_buffers_grow(built, grow):
    import torch
    w = W.AnmlWriter("two")
    w.ste("a", [ord("a")], ["b"], start="all-input", report=True)
    w.ste("b", [ord("b")], report=True)
    groups = nb.Groups(nb.Nfa.from_string(w.text()), group_num=1)
    tables = nb.Tables(groups, precompute_depth=2)
    ts = nb.TableSet([tables])
    rng = np.random.default_rng(3)
    data = rng.choice(np.frombuffer(b"abcd", np.uint8), size=12_000).astype(np.uint8)
    offs, lens = np.array([0, 5000]), np.array([5000, 7000])
    want = [oracle.match(groups.views(), data[o:o + n], 1, int(n))[0] for o, n in zip(offs, lens)]
    assert 1024 < sum(map(len, want)) < CAP  # more than the engine leaves in pinned memory
    dev = torch.from_numpy(data).cuda()
    engine = nb.Engine(0)

    def replay():
        nb.batch_match_async(engine, ts, dev, offs, lens, [0, 0], use_graph=True, result_capacity=CAP)
        engine.sync()
        got = nb.split_by_stream(*nb.batch_results(engine), 2)
        assert all(np.array_equal(g, x) for g, x in zip(got, want))

    replay()
    replay()
    held = engine.memory()["reports"]
    if grow == "sort":  # a standalone sort of more keys than the batch's capacity
        keys = torch.from_numpy(rng.integers(0, 1 << 40, 50 * CAP)).cuda()
        out = torch.empty_like(keys)
        assert engine.sort_unique_device(keys.data_ptr(), len(keys), out.data_ptr()) > 0
    elif grow == "capacity":
        nb.batch_match_async(engine, ts, dev, offs, lens, [0, 0], result_capacity=50 * CAP)
        engine.sync()
    elif grow == "streams":  # a longer batch in between
        many = np.zeros(3000, np.int64)
        nb.batch_match_async(engine, ts, data, many, many + 100, many, result_capacity=50 * CAP)
        engine.sync()
    else:
        engine.match(tables, data, 1, len(data), result_capacity=50 * CAP)
    assert engine.memory()["reports"] > held
    # what the batch's old addresses may hold now
    junk = [torch.full((CAP,), -1, dtype=torch.int64, device="cuda") for _ in range(8)]
    replay()
    replay()
    assert all(bool((j == -1).all()) for j in junk)
