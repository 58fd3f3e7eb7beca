"""The rules that pick a kernel, at their borders (no GPU)."""
import pytest

from tau_rs_b200.csrc import kernels


@pytest.mark.parametrize("experts, width, inner, least", [(64, 2048, 1408, 36), (64, 1024, 704, 48), (8, 512, 1024, 48), (256, 2048, 512, 128), (512, 2048, 512, 256), (4, 256, 256, 96),
                                                          (128, 256, 256, 256)])
def test_experts_are_streamed_once_where_pairs_share_them(experts, width, inner, least):
    """A step of 8 tokens of 6 of 64 large experts is; experts that hardly two pairs share, or whose weights are small, are not."""
    assert kernels.moe_stream_wins(least, experts, width, inner) and not kernels.moe_stream_wins(least - 1, experts, width, inner)
