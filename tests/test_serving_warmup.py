"""A server's warm-up batches are as long as its longest batch, to the byte, so
that what an engine reserves for them is the most that it will need."""
import numpy as np
import pytest

from ngap_b200 import serving as sv


class Slot:
    def __init__(self):
        self.batches = []

    def memory(self):
        return {"input": 0, "reports": 0, "scratch": 0, "plan": 0}

    def launch(self, batch, params):
        self.batches.append([len(r.data) for r in batch])

    def finish(self, nreq):
        return [np.zeros(0, np.int64)] * nreq, 0.0, 0


@pytest.mark.parametrize("most,requests", [(1000, 4), (1003, 4), (1 << 20, 256), ((1 << 20) + 255, 256)])
def test_warmup_batches_are_the_longest(most, requests):
    slot = Slot()
    sv.Server(None, slots=1, budget=1 << 30, max_batch_bytes=most, max_batch_requests=requests,
              slot_factory=lambda i: slot, tables_bytes=0)
    assert [len(b) for b in slot.batches] == [1, requests]
    assert [sum(b) for b in slot.batches] == [most, most]
