"""Rules that pick a kernel's form by sizes alone."""
import pytest
import torch

from questwend_b200.kernels import ops


@pytest.mark.parametrize("lens, heads, key_dim, vdim, tiles", [
    ([4096], 4, 256, 512, True), ([1024] * 4, 4, 256, 512, True), ([700] * 4, 8, 512, 256, True), ([512] * 4, 8, 512, 256, False), ([1000], 4, 256, 512, False),
    ([4096], 16, 128, 128, False), ([2048] + [1] * 16, 4, 256, 512, False), ([4096] + [1] * 63, 8, 512, 256, False), ([130] * 16, 4, 256, 512, False),
    ([256] * 8, 8, 512, 256, False)])
def test_matrix_memory_takes_long_chunks_only_where_they_are_filled(lens, heads, key_dim, vdim, tiles):
    assert ops.mlstm_tiles_pay(sum(lens), len(lens), heads, key_dim, vdim) is tiles


def test_latent_prompts_refuse_the_same_query_sizes_in_both_forms():
    """Query sizes that are no multiple of 16 are refused by the mma.sync kernel: the tcgen05 one does not take them either."""
    assert ops.latent_prefill_tc_fits(128, 64, 128) and ops.latent_prefill_tc_fits(24, 8, 40) and ops.latent_prefill_tc_fits(8, 8, 8)
    assert not ops.latent_prefill_tc_fits(24, 0, 64) and not ops.latent_prefill_tc_fits(64, 8, 64) and not ops.latent_prefill_tc_fits(128, 64, 136)


@pytest.mark.parametrize("lens, heads, key_dim, vdim, tiles", [
    ([4096], 4, 256, 512, True), ([64], 4, 256, 512, True), ([64] * 8, 4, 256, 512, True), ([2048] + [1] * 63, 4, 256, 512, False), ([100], 16, 128, 128, True),
    ([130] * 16, 16, 128, 128, True), ([64] * 8, 16, 128, 128, False), ([4096], 4, 64, 64, False), ([4096], 15, 128, 128, False)])
def test_matrix_memory_takes_long_chunks_for_large_memories(lens, heads, key_dim, vdim, tiles):
    assert ops._mlstm_tiles(sum(lens), len(lens), heads, key_dim, vdim) is tiles


@pytest.mark.parametrize("tokens, top, experts, shared, dtype, grouped", [
    (128, 6, 64, 2816, torch.bfloat16, False), (129, 1, 256, 0, torch.bfloat16, True), (17, 6, 64, 2816, torch.bfloat16, False), (17, 6, 64, 2812, torch.bfloat16, True),
    (16, 8, 8, 2812, torch.bfloat16, False), (128, 2, 16, 0, torch.bfloat16, False), (128, 2, 15, 0, torch.bfloat16, True), (64, 2, 8, 0, torch.bfloat16, False),
    (200, 6, 64, 0, torch.float32, False)])
def test_experts_are_sorted_only_in_long_steps(tokens, top, experts, shared, dtype, grouped):
    x, up, down = (torch.empty(s, dtype=dtype, device="meta") for s in ((tokens, 64), (experts, 64, 64), (experts, 64, 32)))
    assert ops.moe_grouped_fits(x, up, down, top, shared) is grouped


@pytest.mark.parametrize("sizes, fits", [((2048, 1408, 2816, 6, 64), True), ((8, 8, 0, 16, 1024), True), ((8, 8, 0, 16, 1025), False), ((8, 8, 0, 17, 64), False),
                                         ((8, 8, 0, 0, 64), False), ((8, 8, 0, 1, 0), False), ((12, 8, 0, 1, 4), False), ((8, 12, 0, 1, 4), False), ((8, 8, 4, 1, 4), False)])
def test_experts_are_read_once_for_all_where_the_lists_hold_them(sizes, fits):
    assert ops.moe_stream_fits(*sizes) is fits
