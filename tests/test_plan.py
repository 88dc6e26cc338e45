"""Automatic lengths of pieces (filtered tiles) and units (others): they cover
every position once, spread short inputs over the warps, and give the
oracle's reports."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


def traced(engine, tables, data, num_seg, seg_len, algo):
    engine.set_trace(True)
    try:
        got = engine.match(tables, data, num_seg, seg_len, algorithm=algo)
        return got, engine.unit_trace()
    finally:
        engine.set_trace(False)


@pytest.mark.parametrize("filtered", [True, False])
@pytest.mark.parametrize("num_seg,seg_len", [(1, 127), (1, 130), (3, 1000), (1, 20000), (1, 378879), (1, 378881),
                                             (2, 400001), (1, 1300001)])
def test_auto_lengths(engine, num_seg, seg_len, filtered):
    n = num_seg * seg_len
    if filtered:
        anml, data = W.literal_set(seed=5, n_patterns=20, input_len=n, plant_every=max(40, n // 64))
    else:  # most positions report: a filter would pass too much
        w = W.AnmlWriter("dense")
        w.ste("a", W.PRINTABLE[:60], ["b"], start="all-input", report=True)
        w.ste("b", W.PRINTABLE[:60], report=True)
        anml = w.text()
        data = np.random.default_rng(n).choice(W.PRINTABLE, size=n).astype(np.uint8)
    groups = nb.Groups(nb.Nfa.from_string(anml), group_num=1)
    tables = nb.Tables(groups, precompute_depth=2)
    for algo in ("blockinggroups", "nonblockingpcgroups"):
        got, units = traced(engine, tables, data, num_seg, seg_len, algo)
        want, _ = oracle.match(groups.views(), data, num_seg, seg_len)
        assert np.array_equal(got, want)
        for s in range(num_seg):
            u = np.sort(units[units["stream"] == s], order="lo")
            assert u["lo"][0] == 0 and u["hi"][-1] == seg_len
            assert np.array_equal(u["lo"][1:], u["hi"][:-1])
        longest = int((units["hi"] - units["lo"]).max())
        if filtered and n >= 1 << 17:  # one piece per scan warp (32 per SM), in steps of 512 positions
            assert longest <= min(4096, max(256, -(-n // (148 * 32)) + 511))
        else:  # one unit per warp (16 per SM), or 128 positions where that is longer
            assert longest <= min(2048, max(128, -(-n // (148 * 16)) + 63))
