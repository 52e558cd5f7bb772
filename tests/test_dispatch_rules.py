"""Rules that choose between two ways to the same result, from sizes that the host knows."""
import pytest


@pytest.mark.parametrize("window,max_new,max_total,apart", [
    (None, 1024, 1024, False), (None, 1, 5000, True), (None, 3, 3, True), (None, 4, 9000, False),
    (512, 512, 512, False), (512, 500, 574, False), (512, 500, 575, True), (512, 2048, 2048, True), (1024, 1100, 1100, False),
    (1024, 256, 1256, True), (4096, 256, 1256, False), (16, 1, 4, True)])
def test_tokens_past_a_window_are_worked_one_a_block(window, max_new, max_total, apart):
    from gemmars_b200 import kernels
    assert kernels.attention_tokens_apart(window, max_new, max_total) is apart


def _step(lens, heads, host=True):
    return type("Ctx", (), {"max_new": max(lens), "n_tokens": sum(lens), "n_seqs": len(lens), "extras": {}, "host": {"seq_len": lens} if host else None})()


@pytest.mark.parametrize("form,heads,lens,chunks", [
    ("delta", 16, [64], False), ("delta", 16, [128], True), ("delta", 32, [96], True), ("delta", 16, [32] * 16, True),
    ("channel_delta", 16, [128], False), ("channel_delta", 32, [128], True), ("ssd", 32, [128], False), ("ssd", 32, [192], True),
    ("before", 32, [128], False), ("before", 64, [256], True), ("after", 16, [128], False), ("after", 16, [256], True),
    ("delta", 16, [31] * 64, False),                       # no sequence brings two chunks
    ("delta", 16, [1] * 128 + [128], False), ("delta", 16, [1] * 128 + [512], True), ("delta", 32, [1] * 32 + [64], False),
    ("ssd", 64, [1] * 128 + [512], False), ("delta", 32, [2048], True), ("before", 64, [33] * 16, False), ("before", 64, [64] * 16, True)])
def test_prompts_walk_their_recurrences_in_chunks_where_that_is_faster(form, heads, lens, chunks):
    from gemmars_b200 import kernels
    ctx = _step(lens, heads)
    assert kernels.chunk_scan(form, "bfloat16", 128, heads, ctx) is chunks
    assert kernels.chunk_scan(form, "bfloat16", 128, heads, ctx) is chunks          # with what the step keeps
    assert not kernels.chunk_scan(form, "float32", 128, heads, _step(lens, heads))
    assert not kernels.chunk_scan(form, "bfloat16", 129, heads, _step(lens, heads))
    if len(lens) == 1 and lens[0] % 16 == 0:               # lengths that only the device knows: as many chunks as there can be
        assert kernels.chunk_scan(form, "bfloat16", 128, heads, _step(lens, heads, host=False)) is chunks
