"""Host rules that choose a kernel from a step's sizes (no device needed), at sizes where both sides were timed."""
import pytest

from torchless_rs_b200.csrc.latent_bf16 import prompt_times


@pytest.mark.parametrize("past,new,heads,window,tiles", [
    ([0], [300], 16, 4096, True), ([0], [256], 16, 4096, False), ([0], [2048], 16, 4096, True), ([0], [1000], 16, None, True),
    ([0] * 4, [256] * 4, 16, 4096, True), ([0] * 8, [256] * 8, 16, 4096, False), ([0] * 64, [256] * 64, 16, 4096, False),
    ([0] * 32, [350] * 32, 16, 4096, False), ([0] * 32, [500] * 32, 16, 4096, True), ([256] * 32, [512] * 32, 16, 4096, True),
    ([0] * 33, [512] + [50] * 32, 16, 4096, False), ([0] * 33, [512] + [200] * 32, 16, 4096, False),
    ([0] + [199] * 63, [256] + [200] * 63, 16, 4096, False), ([0] + [100] * 63, [256] + [104] * 63, 16, 4096, False),
    ([0] + [999] * 15, [256] + [1000] * 15, 16, 4096, True), ([0] + [3999] * 7, [256] + [4000] * 7, 16, 4096, True),
    ([0, 7999], [256, 8000], 16, 4096, True), ([0] * 64, [128] * 64, 32, 4096, False), ([0] * 64, [40] * 64, 128, 4096, False),
    ([0], [33], 128, 4096, False), ([1000] * 4, [1033] * 4, 128, 4096, True), ([0] * 32, [600] * 32, 8, 4096, True),
    ([0], [4096], 1, 4096, True)])
def test_latent_attention_of_prompts_runs_where_it_was_faster(past, new, heads, window, tiles):
    here, there = prompt_times(past, new, heads, window, 148)
    assert (here < there) == tiles, (here, there)
