"""Automatic chunk lengths: units of a bounded tile cover every position once,
at most one per resident warp for short inputs, and give the oracle's reports."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_seg,seg_len", [(1, 127), (1, 129), (3, 1000), (1, 378879), (1, 378881),
                                             (2, 400001)])
def test_auto_chunks(engine, num_seg, seg_len):
    n = num_seg * seg_len
    anml, data = W.literal_set(seed=5, n_patterns=20, input_len=n, plant_every=max(40, n // 64))
    groups = nb.Groups(nb.Nfa.from_string(anml), group_num=1)
    tables = nb.Tables(groups, precompute_depth=2)
    for algo in ("blockinggroups", "nonblockingpcgroups"):
        engine.set_trace(True)
        try:
            got = engine.match(tables, data, num_seg, seg_len, algorithm=algo)
            units = engine.unit_trace()
        finally:
            engine.set_trace(False)
        want, _ = oracle.match(groups.views(), data, num_seg, seg_len)
        assert np.array_equal(got, want)
        for s in range(num_seg):
            u = np.sort(units[units["stream"] == s], order="lo")
            assert u["lo"][0] == 0 and u["hi"][-1] == seg_len
            assert np.array_equal(u["lo"][1:], u["hi"][:-1])
        longest = int((units["hi"] - units["lo"]).max())
        assert longest <= 2048
        # one unit per warp of a full grid (16 per SM), or 128 positions where that is longer
        warps = 148 * 16
        assert longest <= max(128, -(-n // warps) + 63)
