"""Device input read in place (address and length multiples of 16) or copied:
every alignment gives the oracle's reports, and nothing past the input counts."""
import numpy as np
import pytest

import ngap_b200 as nb
from ngap_b200 import workloads as W
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", [0, 1, 8, 16, 48])
@pytest.mark.parametrize("length", [16, 4096, 4097, 200_000, 200_016])
def test_device_input(engine, start, length):
    import torch
    anml, data = W.literal_set(seed=5, n_patterns=20, input_len=length, plant_every=max(20, length // 64))
    groups = nb.Groups(nb.Nfa.from_string(anml), group_num=1)
    tables = nb.Tables(groups, precompute_depth=2)
    want, _ = oracle.match(groups.views(), data, 1, length)
    # what follows the input would match: copies of its planted patterns
    buf = torch.from_numpy(np.concatenate([np.resize(data[::-1], start), data, data[:64]]).astype(np.uint8)).cuda()
    got = engine.match(tables, buf[start:start + length], 1, length)
    assert np.array_equal(got, want)
    nb.batch_match_async(engine, nb.TableSet([tables]), buf[start:start + length], [0], [length], [0])
    engine.sync()
    assert np.array_equal(nb.batch_results(engine)[0], want)
    # a temporary tensor on a stream of its own stays alive until the match ends
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        engine.match_async(tables, buf[start:start + length].clone(), 1, length, stream=side.cuda_stream)
        junk = torch.full((length,), 65, dtype=torch.uint8, device="cuda")
    engine.sync()
    assert np.array_equal(engine.results(), want)
    del junk


@pytest.mark.parametrize("length", [2**31 + 4099, 2**32 - 16, 2**32 - 1])
def test_largest_input(built, length):
    """Segments past 2 GiB and up to the end of the 32-bit offsets: text planted
    at both ends, across a piece's and a scan launch's edges and past 2 GiB
    gives the oracle's reports of it, moved to its place."""
    import torch
    anml, text = W.literal_set(seed=6, n_patterns=20, input_len=600, plant_every=40)
    groups = nb.Groups(nb.Nfa.from_string(anml), group_num=1)
    tables = nb.Tables(groups, precompute_depth=2)
    found, _ = oracle.match(groups.views(), text, 1, len(text))
    assert len(found) > 0
    buf = torch.zeros(length, dtype=torch.uint8, device="cuda")
    places = [0, 4096 * 3 - 300, (32 << 20) - 300, 2**31 + 7, length - len(text)]
    for at in places:
        buf[at:at + len(text)] = torch.from_numpy(text)
    want = np.sort(np.concatenate([found + np.uint64(at) for at in places]))
    engine = nb.Engine(0)
    got = engine.match(tables, buf, 1, length)
    assert np.array_equal(np.sort(got), want)
