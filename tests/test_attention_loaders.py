"""The barrier model of test_attention_protocol.py with the loads in the order in which
fa_fwd_sm100.cu issues them: the next item's first K ahead of its Q, whose buffers are still
being read when that K already has a ring slot."""
import random

import pytest

from test_attention_protocol import Kernel, _item_lists


class FirstKeyAhead(Kernel):
    def loader(self):
        it = 0

        def kv_load():
            nonlocal it
            s, n = it % self.slots, it // self.slots
            if n > 0:
                yield from self.wait(self.kv_free[s], n - 1)
            self.tma.append(("kv", s, None, self.kv_full[s]))
            it += 1

        for i, (nt0, nt1) in enumerate(self.items):
            yield from kv_load()
            for s in range(2):
                if i > 0:
                    yield from self.wait(self.q_free[s], i - 1)
                self.tma.append(("q", s, i, self.q_full[s]))
            for j in range(nt1):
                yield from kv_load()
                if j + 1 < nt1:
                    yield from kv_load()
            yield


@pytest.mark.parametrize("slots,stream", [(5, True), (8, False)])
@pytest.mark.parametrize("causal", [False, True])
def test_loads_hold_under_random_interleavings(slots, stream, causal):
    for items in _item_lists(causal):
        for seed in range(8):
            FirstKeyAhead(items, slots, stream, causal, random.Random(seed)).run()
            if seed < 4:
                FirstKeyAhead(items, slots, stream, causal, random.Random(1000 + seed)).run(skew=True)
