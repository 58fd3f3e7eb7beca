"""The rules that pick a kernel, at their borders (no GPU)."""
import pytest

from tau_rs_b200.csrc import kernels


@pytest.mark.parametrize("experts, width, inner, least", [(64, 2048, 1408, 36), (64, 1024, 704, 48), (8, 512, 1024, 48), (256, 2048, 512, 128), (512, 2048, 512, 256), (4, 256, 256, 96),
                                                          (128, 256, 256, 256)])
def test_experts_are_streamed_once_where_pairs_share_them(experts, width, inner, least):
    """A step of 8 tokens of 6 of 64 large experts is; experts that hardly two pairs share, or whose weights are small, are not."""
    assert kernels.moe_stream_wins(least, experts, width, inner) and not kernels.moe_stream_wins(least - 1, experts, width, inner)


@pytest.mark.parametrize("n_seqs, tokens, max_len, n_heads, tiled", [(1, 20, 64, 16, True), (1, 20, 65, 16, False), (1, 777, 777, 16, False), (16, 320, 128, 16, True), (16, 320, 129, 16, False),
                                                                     (15, 300, 128, 16, False), (16, 1600, 102, 16, False), (200, 4000, 192, 8, True), (200, 4000, 193, 8, False), (65, 164, 2001, 16, False)])
def test_float32_runs_by_their_number_and_contexts(n_seqs, tokens, max_len, n_heads, tiled):
    """Contexts of one page, and many short runs over two or three, stay on the 32-bit pipes."""
    assert kernels.tiled_attention_wins(n_seqs, tokens, max_len, n_heads) == tiled
