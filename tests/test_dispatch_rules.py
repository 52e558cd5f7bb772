"""Rules that choose between two ways to the same result, from sizes that the host knows."""
import pytest


@pytest.mark.parametrize("window,max_new,max_total,apart", [
    (None, 1024, 1024, False), (None, 1, 5000, True), (None, 3, 3, True), (None, 4, 9000, False),
    (512, 512, 512, False), (512, 500, 574, False), (512, 500, 575, True), (512, 2048, 2048, True), (1024, 1100, 1100, False),
    (1024, 256, 1256, True), (4096, 256, 1256, False), (16, 1, 4, True)])
def test_tokens_past_a_window_are_worked_one_a_block(window, max_new, max_total, apart):
    from gemmars_b200 import kernels
    assert kernels.attention_tokens_apart(window, max_new, max_total) is apart
