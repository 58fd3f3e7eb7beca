"""Attention over cached latent rows on the tensor cores, at the sizes where it can go wrong, against 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, rank, rot", [(16, 512, 64), (1, 64, 32), (17, 128, 0), (33, 448, 64), (8, 512, 128), (5, 192, 96)])
@pytest.mark.parametrize("window, splits", [(0, 1), (0, 3), (70, 1), (70, 5)])
def test_tensor_core_kernel(heads, rank, rot, window, splits):
    """Heads around a block's 16, latents of one to eight tiles a warp, contexts around its 64 rows, ranges that are empty, a window that begins inside
    a page, sinks, an infinity behind the end of a sequence."""
    torch.manual_seed(heads + rank)
    lengths, width = [1, 63, 64, 65, 130, 300], rank + rot
    stride = 5
    pages = torch.randn(len(lengths) * stride, 64, width, device="cuda").to(torch.bfloat16)
    table = torch.randperm(len(lengths) * stride).view(len(lengths), stride).to(torch.int32).cuda()
    for index, length in enumerate(lengths):
        if length % 64:
            pages[int(table[index, length // 64]), length % 64 :] = float("inf")
    queries = torch.randn(len(lengths), heads, width, device="cuda").to(torch.bfloat16)
    sinks = torch.randn(heads, device="cuda")
    positions = torch.tensor([length - 1 for length in lengths], dtype=torch.int32).cuda()
    sequence = torch.arange(len(lengths), dtype=torch.int32).cuda()
    found = torch.full((len(lengths), heads, rank), float("nan"), device="cuda", dtype=torch.bfloat16)
    scale = width ** -0.5
    kernels.latent_attention(queries, pages, found, sinks, positions, sequence, table, heads, rank, rot, scale, window, splits)
    for index, length in enumerate(lengths):
        rows = pages[table[index].long()].reshape(-1, width)[:length].double()[max(0, length - window) if window else 0 :]
        scores = queries[index].double() @ rows.T * scale
        weights = torch.softmax(torch.cat([scores, sinks.double()[:, None]], dim=1), dim=1)[:, :-1]
        wanted = weights @ rows[:, :rank]
        # One bfloat16 rounding of the result, beside 32-bit sums.
        assert bool(((found[index].double() - wanted).abs() <= 2.0 ** -8 * wanted.abs() + 1e-5).all()), (index, float((found[index].double() - wanted).abs().max()))
