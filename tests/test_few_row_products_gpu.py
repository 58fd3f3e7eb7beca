"""Products of a batch of heads over few rows, at the sizes where their kernel changes, against 64-bit."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows, batch, features, depth", [(1, 1, 1, 8), (8, 16, 512, 128), (9, 16, 512, 128), (8, 17, 512, 128), (16, 33, 130, 512), (3, 3, 77, 1000)])
def test_blocks_up_to_512_and_more(dtype, rows, batch, features, depth):
    """Blocks that load ahead of the kernel in front and blocks that do not, features and columns cut anywhere, rows inside wider ones."""
    torch.manual_seed(features)
    values, weight = torch.randn(rows, batch, depth + 8, device="cuda").to(dtype)[:, :, :depth], torch.randn(batch, features, depth, device="cuda").to(dtype)
    out = torch.full((rows, batch, features + 3), 7.0, device="cuda")      # 32-bit results of either type
    kernels.gemm_simt_batched(values, weight, out[:, :, :features])
    wanted = torch.einsum("mbk,bnk->mbn", values.double(), weight.double())
    magnitude = torch.einsum("mbk,bnk->mbn", values.double().abs(), weight.double().abs())
    # A rounding for every term of a lane's chain, and for the sums that join the lanes.
    assert bool(((out[:, :, :features].double() - wanted).abs() <= (depth + 5) * 2.0 ** -24 * magnitude).all()) and bool((out[:, :, features:] == 7.0).all())
