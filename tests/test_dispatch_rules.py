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


def _walked(window, lens, starts, tokens):
    """What attention_ref.cu's blocks walk, token by token."""
    where = [(i, s + j) for i, (n, s) in enumerate(zip(lens, starts)) for j in range(n)]
    blocks = []
    for a in range(0, len(where), tokens):
        keys, t, block = 0, 0, where[a:a + tokens]
        first = [max(0, p + 1 - window) if window else 0 for _, p in block]
        while t < len(block):
            end = t
            while end < len(block) and block[end][0] == block[t][0] and first[end] == first[t]:
                end += 1
            keys += block[end - 1][1] + 1 - first[t]
            t = end
        blocks.append(keys)
    return max(blocks), sum(blocks)


@pytest.mark.parametrize("tokens", [1, 4, 8, 16])
def test_the_keys_that_blocks_of_the_plain_attention_walk(tokens):
    import random
    from gemmars_b200 import kernels
    rng = random.Random(tokens)
    for _ in range(300):
        n = rng.randint(1, 12)
        lens = [rng.choice((1, 1, 2, 5, rng.randint(1, 90))) for _ in range(n)]
        starts = [rng.choice((0, 0, rng.randint(1, 200))) for _ in range(n)]
        window = rng.choice((None, 1, 3, 40, 64, 1000))
        assert kernels.attention_ref_passes(window, lens, starts, tokens) == _walked(window, lens, starts, tokens)


@pytest.mark.parametrize("nh,nkv,lens,starts,window,forms", [
    # prompts alone, both sides of the lines by size
    (16, 8, [144], [0], None, (1,)), (16, 8, [145], [0], None, (16,)), (16, 8, [75, 90, 136], [0] * 3, None, (16,)), (8, 8, [288], [0], None, (4,)),
    (8, 8, [289], [0], None, (16,)), (8, 8, [147], [0], None, (1,)), (32, 8, [72], [0], None, (1,)), (32, 8, [73], [0], None, (16,)),
    # beside single tokens of long conversations
    (16, 8, [301] + [1] * 8, [0] + [2000] * 8, None, (1,)), (16, 8, [301] + [1] * 16, [0] + [8000] * 16, None, (1,)),
    (16, 8, [1024] + [1] * 16, [0] + [2000] * 16, None, (1,)), (16, 8, [1024] + [1] * 40, [0] + [500] * 40, None, (16,)),
    (16, 16, [1024] + [1] * 8, [0] + [2000] * 8, None, (4,)), (16, 16, [1024] + [1] * 40, [0] + [500] * 40, None, (4,)),
    (16, 16, [1024] + [1] * 16, [0] + [8000] * 16, None, (1,)), (32, 8, [1024] + [1] * 16, [0] + [2000] * 16, None, (1,)),
    (32, 8, [1024] + [1] * 40, [0] + [500] * 40, None, (16,)),
    # past a window
    (16, 8, [528], [0], 512, (1,)), (16, 8, [700], [0], 512, (1,)), (16, 16, [528], [0], 512, (4,)), (16, 16, [2098], [0], 2048, (4,)),
    (16, 8, [2098], [0], 2048, (4, 16)), (16, 8, [512], [0], 512, (16,)), (16, 16, [512, 586], [0, 0], 512, (4,)), (32, 8, [512, 586], [0, 0], 512, (16,)),
    # a few tokens each
    (16, 8, [7] * 30, [500] * 30, None, (16,)), (16, 16, [5] * 60, [100] * 60, None, (4,)), (16, 8, [3] * 100, [500] * 100, None, (1,))])
def test_the_plain_attention_takes_the_form_that_was_the_fastest(nh, nkv, lens, starts, window, forms):
    from gemmars_b200 import kernels
    assert kernels.attention_ref_form(window, lens, starts, nh, nkv, 128) in forms


def test_heads_too_wide_for_sixteen_queries_take_four_tokens():
    from gemmars_b200 import kernels
    assert kernels.attention_ref_form(None, [300], [0], 16, 8, 200) == 4 and kernels.attention_ref_form(None, [100], [0], 16, 8, 200) == 1


def test_heads_that_the_plain_attention_refuses_are_left_to_it():
    from gemmars_b200 import kernels
    assert [kernels.attention_ref_form(None, [500], [0], nh, nkv, 64) for nh, nkv in ((2, 4), (6, 4))] == [1, 1]
