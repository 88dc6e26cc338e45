"""Units of cyclic rules: several tiles by many segments, fewer units than CTAs,
fewer than warps, and more (first units by number, later ones from the cursor)."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu

LOWER = np.frombuffer(b"abcdefghij", np.uint8)


@pytest.fixture(scope="module")
def groups(built):
    rng = np.random.default_rng(8)
    w = W.AnmlWriter("loops")
    for n in range(120):  # ab+cd, some with a .* that another follows
        a = rng.choice(LOWER, 4).tolist()
        for i in range(4):
            w.ste(f"r{n}_{i}", [a[i]], ([f"r{n}_{i}"] if i == 1 else []) + ([f"r{n}_{i + 1}"] if i < 3 else []),
                  start="all-input" if i == 0 else None, report=i == 3)
    for n in range(8):
        for p in range(3):
            w.ste(f"x{n}_{p}", [int(rng.choice(LOWER))], [f"s{n}_{p}", f"x{n}_{p + 1}"] if p < 2 else [],
                  start="all-input" if p == 0 else None, report=p == 2)
            if p < 2:
                w.ste(f"s{n}_{p}", None, [f"s{n}_{p}", f"x{n}_{p + 1}"], symbol_set="*")
    g = nb.Groups(nb.Nfa.from_string(w.text()), group_num=3)
    assert sum(t["max_path"] < 0 for t in g.tiles(precompute_depth=-1)) >= 3
    return g


@pytest.mark.parametrize("num_seg,seg_len", [(1, 3000), (40, 500), (300, 90), (1500, 40), (5000, 17)])
@pytest.mark.parametrize("depth,algorithm", [(-1, "nonblockingpcgroups"), (0, "NAPgroups"), (0, "blockinggroups")])
def test_units(engine, groups, num_seg, seg_len, depth, algorithm):
    tables = nb.Tables(groups, precompute_depth=depth)
    data = np.random.default_rng(num_seg).choice(LOWER, num_seg * seg_len).astype(np.uint8)
    want, _ = oracle.match(groups.views(), data, num_seg, seg_len)
    for unique in (False, True):
        got = engine.match(tables, data, num_seg, seg_len, algorithm=algorithm, unique=unique)
        assert len(want) > 0 and np.array_equal(got, want)
    engine.set_trace(True)
    try:
        engine.match(tables, data, num_seg, seg_len, algorithm=algorithm)
        u = engine.unit_trace()
    finally:
        engine.set_trace(False)
    assert len(u) >= 3 * num_seg and np.all(u["cycles"] > 0)  # every unit ran
