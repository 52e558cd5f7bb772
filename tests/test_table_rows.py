"""Page table rows that go out with a step's index block arrive as a copy of the whole table would have them."""
import numpy as np
import pytest
import torch

from gemmars_b200.cache.pool import KVNeed, SequenceCache


@pytest.mark.parametrize("slots", [1, 2, 3, 7])
def test_rows_put_are_the_rows_synced(slots):
    cache = SequenceCache([(0, [KVNeed(2, 16)]), (1, [KVNeed(2, 16, window=100)])], 4096, slots, 0, 64, torch.float32, torch.device("cpu"))
    held = [cache.open() for _ in range(slots)]
    for step, new in enumerate((70, 1, 200)):
        for i, s in enumerate(held):
            cache.extend(s, new + i)
        if step == 1:
            cache.close(held[0])
            held[0] = cache.open()
        assert cache.changed() == (sum(len(g.changed_rows()) for g in cache.kv_groups),
                                   sum(g.table_rows(g.changed_rows()).size for g in cache.kv_groups))
        for g in cache.kv_groups:
            rows = g.changed_rows()
            values = torch.from_numpy(g.table_rows(rows).astype(np.int32))
            g.put_rows(rows, values)
            assert torch.equal(g.page_table, g.table_host)
        assert cache.changed() == (0, 0)
        cache.sync()                       # nothing is left to send
        for g in cache.kv_groups:
            assert torch.equal(g.page_table, g.table_host)
