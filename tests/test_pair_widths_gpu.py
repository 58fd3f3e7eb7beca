"""Products on pairs of SMs in tiles of other widths than 256."""
import pytest
import torch

from tau_rs_b200.csrc import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [64, 96, 128, 160, 192, 224])
@pytest.mark.parametrize("m, n, k, dtype, gated", [(129, 16, 64, torch.bfloat16, False), (300, 1000, 200, torch.bfloat16, False), (257, 20004, 72, torch.float32, False),
                                                   (513, 4096 + 48, 136, torch.bfloat16, True), (200, 332, 1032, torch.float32, False)])
def test_any_width(width, m, n, k, dtype, gated):
    """Widths that cut passes of 128, 64 and 32 features and tiles that cut the features anywhere, more tiles than pairs, rows that do not start on 16 bytes: what tiles of 256 leave,
    bit for bit (the same sums), beside columns that stay."""
    torch.manual_seed(k)
    x, w = torch.randn(m, k, device="cuda").to(torch.bfloat16), torch.randn(n, k, device="cuda").mul(k ** -0.5).to(torch.bfloat16)
    bias = None if gated else torch.randn(n, device="cuda")
    columns = n // 2 if gated else n
    results = []
    for features in (256, width):
        wide = torch.full((m, columns + 16), 7.0, device="cuda", dtype=dtype)
        out = wide[:, 8 : 8 + columns] if features != width or width % 64 else wide[:, 1 : 1 + columns]      # odd rows are stored one by one
        kernels.gemm_tc(x, w, bias, out, 256, gated, 0, 1, pair_width=features)
        assert bool((wide[:, columns + 8 :] == 7.0).all()) and bool((wide[:, :1] == 7.0).all())
        results.append(out.clone())
    assert torch.equal(*results)
    if not gated:
        wanted = x.double() @ w.double().T + bias.double()
        assert float((results[1].double() - wanted).abs().max() / wanted.abs().max()) < (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)
    assert kernels.build.load_library("gemm_tc.cu").tau_gemm_tc_status() == 0


@pytest.mark.parametrize("m, n, k, pairs", [(129, 64, 2048, False), (160, 512, 2048, False), (129, 1024, 2048, False), (200, 1024, 2048, True), (129, 2048, 2048, True), (257, 512, 2048, True)])
def test_few_tiles_are_cut_along_k_or_go_to_pairs(m, n, k, pairs):
    """At the border between them: the bits of 32-bit results tell one order of sums from the other."""
    torch.manual_seed(n)
    x, w = torch.randn(m, k, device="cuda").to(torch.bfloat16), torch.randn(n, k, device="cuda").to(torch.bfloat16)
    picked, paired, cut = (torch.empty(m, n, device="cuda") for _ in range(3))
    kernels.gemm_tc(x, w, None, picked)
    kernels.gemm_tc(x, w, None, paired, 256, pair=1)
    kernels.gemm_tc(x, w, None, cut, 256, pair=0)
    assert not torch.equal(paired, cut) and torch.equal(picked, paired if pairs else cut)
