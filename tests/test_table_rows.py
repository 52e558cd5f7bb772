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


@pytest.mark.gpu
@pytest.mark.parametrize("slots", [1, 5, 16, 40])
def test_rows_put_on_the_device_take_a_launch_a_group(slots):
    from gemmars_b200 import kernels
    dev = torch.device("cuda")
    cache = SequenceCache([(0, [KVNeed(2, 16)]), (1, [KVNeed(2, 16, window=100)])], 16384, slots, 0, 64, torch.float32, dev)
    held = [cache.open() for _ in range(slots)]
    for new in (70, 1, 100):
        for i, s in enumerate(held):
            cache.extend(s, new + i)
        before = kernels.launch_count()
        sent = 0
        for g in cache.kv_groups:
            rows = g.changed_rows()
            sent += bool(len(rows))
            g.put_rows(rows, torch.from_numpy(g.table_rows(rows).astype(np.int32)).to(dev), torch.from_numpy(rows.astype(np.int32)).to(dev))
            assert torch.equal(g.page_table.cpu(), g.table_host)
        assert kernels.launch_count() - before == sent
        assert cache.changed() == (0, 0)


@pytest.mark.gpu
def test_a_prompt_step_sends_its_rows_with_its_index_block(model_folders, monkeypatch):
    """However many sequences start in it: nothing of the page table is copied apart, and no row by itself."""
    import plain_qwen3 as plain
    from tiny_configs import TINY_B

    from gemmars_b200 import Engine
    from gemmars_b200.cache.pool import KVGroup
    from gemmars_b200.engine.step import StepItem
    folder = model_folders(TINY_B)
    pcfg, w = plain.load_folder(folder)
    runner = Engine.load(folder, "dtype=float32;max_batch=24;max_tokens=4096").runner
    put, sent = KVGroup.put_rows, []

    def watched(self, rows, values, *at):
        sent.append((len(rows), len(at)))
        put(self, rows, values, *at)
    monkeypatch.setattr(KVGroup, "put_rows", watched)
    monkeypatch.setattr(KVGroup, "sync", lambda self: pytest.fail("a copy of its own"))
    rng = np.random.default_rng(1)
    prompts = [rng.integers(0, TINY_B["vocab_size"], 5 + i).tolist() for i in range(24)]
    out = runner.step([StepItem(runner.open(), t, [len(t) - 1]) for t in prompts])
    assert sent == [(24, 1)] * len(runner.cache.kv_groups)
    for i in (0, 23):
        want = np.asarray(plain.forward(pcfg, w, prompts[i]))[-1]
        assert np.abs(out[i].double().cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()


@pytest.mark.gpu
def test_the_largest_step_pins_no_new_memory(model_folders):
    """As many tokens as a step takes, every one's logits wanted, and page table rows beside them."""
    from tiny_configs import TINY_C

    from gemmars_b200 import Engine
    from gemmars_b200.engine.step import Runner, StepItem
    model = Engine.load(model_folders(TINY_C), "dtype=float32;max_batch=8;max_tokens=512").runner.model
    runner = Runner(model, 8192, max_batch=8, prefill_chunk=256, max_step_tokens=256)
    pinned = [b.data_ptr() for b in runner._ring.bufs]
    rng = np.random.default_rng(1)
    for lens in ((200, 56), (32,) * 8, (256,)):
        slots = [runner.open() for _ in lens]
        assert sum(runner.cache.changed()) <= runner.max_step_tokens
        runner.step([StepItem(s, rng.integers(0, 301, n).tolist(), list(range(n))) for s, n in zip(slots, lens)])
        for s in slots:
            runner.close(s)
    assert [b.data_ptr() for b in runner._ring.bufs] == pinned
