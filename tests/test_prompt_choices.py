"""Host rules that choose a kernel from a step's sizes (no device needed), at sizes where both sides were timed."""
import pytest

from torchless_rs_b200.csrc import attention_f32, latent_bf16


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
    here, there = latent_bf16.prompt_times(past, new, heads, window, 148)
    assert (here < there) == tiles, (here, there)


@pytest.mark.parametrize("past,new,nh,nkv,hd,window,tiles", [
    ([2000], [2002], 32, 8, 128, None, False), ([2000], [2008], 32, 8, 128, None, True), ([8000], [8004], 32, 8, 128, None, False),
    ([500], [508], 32, 8, 128, None, True), ([500], [504], 32, 8, 128, None, False), ([100], [108], 32, 8, 128, None, False),
    ([100], [116], 32, 8, 128, None, True), ([0], [400], 32, 8, 128, None, True), ([0, 0], [400, 131], 32, 8, 128, None, True),
    ([0], [42], 32, 8, 128, None, True), ([0] * 64, [5] * 64, 32, 8, 128, None, False), ([100] * 64, [102] * 64, 32, 8, 128, None, True),
    ([999] * 4, [1000] * 3 + [1001], 32, 8, 128, None, True), ([3999, 3998], [4000, 4000], 32, 8, 128, None, False),
    ([100] * 64, [102] * 64, 32, 32, 128, None, False), ([0] * 16, [64] * 16, 32, 32, 128, None, True),
    ([2000], [2008], 32, 8, 128, 200, False), ([2000], [2016], 32, 8, 128, 200, True),
    ([500], [508], 16, 4, 64, None, False), ([500], [532], 16, 4, 64, None, True), ([2000], [2064], 64, 8, 64, None, True),
    ([500], [502], 8, 8, 32, None, True), ([0] * 64, [5] * 64, 8, 8, 32, None, False), ([2000], [2002], 4, 2, 16, None, True),
    ([500], [564], 4, 2, 16, 200, False), ([500], [628], 32, 8, 16, 200, True)])
def test_32_bit_prompt_attention_runs_where_it_was_faster(past, new, nh, nkv, hd, window, tiles):
    in_tiles, by_rows = attention_f32.prompt_times(past, new, nh, nkv, hd, window, 148)
    assert (in_tiles < by_rows) == tiles, (in_tiles, by_rows)


@pytest.mark.parametrize("past,new,decode,formed", [
    ([0], [511], False, False), ([0], [512], False, True), ([0] * 300, [600] + [1] * 299, False, False),
    ([0] * 100, [600] + [1] * 99, False, True), ([0, 1], [700, 9], False, False), ([0], [512], True, False), ([0] * 2, [1, 900], False, True)])
def test_latent_attention_forms_keys_for_long_steps_that_start_their_sequences(past, new, decode, formed):
    from types import SimpleNamespace
    assert latent_bf16.LatentPrompt.takes(SimpleNamespace(is_decode=decode, past_lens=past, new_lens=new)) == formed
    assert not latent_bf16.LatentPrompt.takes(SimpleNamespace(is_decode=False))     # a step whose lengths nobody says


@pytest.mark.parametrize("new,window,formed", [
    ([512] + [1] * 127, None, False), ([600] + [1] * 99, None, True), ([600] + [1] * 99, 64, False), ([600] + [1] * 99, 600, True),
    ([2048] + [1] * 200, 256, False), ([2048] + [1] * 200, 4096, True), ([600] + [14] * 60, 64, True), ([2048], 1, True)])
def test_latent_attention_forms_keys_of_many_short_sequences_only_where_that_was_faster(new, window, formed):
    """A sequence of a few tokens costs its block here what one of 128 costs, and with a window the other kernels have little to do."""
    from types import SimpleNamespace
    step = SimpleNamespace(is_decode=False, past_lens=[0] * len(new), new_lens=new)
    assert latent_bf16.LatentPrompt.takes(step, window) == formed
