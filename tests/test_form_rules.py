"""Rules that pick a kernel's form by sizes alone."""
import pytest

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
